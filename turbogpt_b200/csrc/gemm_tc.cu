// BF16 GEMM on the 5th-generation tensor cores: C[m,n] = sum_k A[m,k] * B[n,k], FP32
// accumulation in tensor memory.  Replaces the reference's warp-level mma.sync products
// (cuda/mma.cuh:69-108, cuda/ops.cuh:30-55,83-117) for every projection, input-gradient and
// weight-gradient GEMM of the step.
//
// One persistent CTA per SM (or one CTA pair per two SMs, cta_group::2, for 256-row tiles) walks
// output tiles of 128 x BN (BN = 64..256).  Warp 0 streams operand slices of 64 K-elements with
// TMA into a ring of 128-byte-swizzled shared-memory stages; warp 1 issues tcgen05.mma (one
// thread) into one of two 256-column TMEM accumulators; sixteen epilogue warps drain the other
// accumulator, so the epilogue of tile i overlaps the main loop of tile i+1.  Either operand may be
// K-major (row = 64 contiguous K elements) or MN-major (row = 64 contiguous M/N elements for one K
// index), which covers y = x W^T, dx = dy W and dW = dy^T x on row-major tensors without transposes.
//
// Epilogue: four warps share each 32-lane quarter of tensor memory and take every fourth
// 32-column chunk.  A lane reads its row's accumulator chunk (tcgen05.ld), exchanges half of it with its neighbour (so that a
// 256-bit access covers 16 rows instead of 32), optionally combines it with the same part of a second tensor read straight from global
// memory one chunk ahead (residual, saved GELU derivative, or the Newton-Schulz operand), and stores.  Over a short K the epilogue
// is as long as the products or longer: clocks of a 128 x 256 tile inside the 12-layer step, where K 768 takes the tensor pipe 6144: GELU with
// its derivative 8000 (11700 with a lane to a row, one value at a time, and a pair's warps awaiting their stores), GELU gradient
// 7500 (11800), plain 3100 (7200).  Over a long K the products take their 512 clocks a 64-deep block of a 256 x 256 tile (8192^3: 513).
//
// Weight-gradient GEMMs have few output tiles and a very long K; they are split along K and each
// split writes an FP32 partial tile to a workspace.  With two or three splits the last one to finish
// a tile (an atomic ticket, no spinning) sums the partials in split order; with four or more a second
// kernel adds them, in the same order, over the whole GPU.  Results are deterministic either way.
// The head GEMM has an epilogue of its own: 256-way softmax cross-entropy on the FP32 accumulators.
#include "device_utils.cuh"
#include "sm100.cuh"
#include "tile_rows.cuh"
#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <atomic>
#include <mutex>
#include <type_traits>
#include <unordered_map>

using namespace sm100;

namespace {
constexpr int BM = 128, BK = 64, MaxBN = 256, MaxStages = 8;
constexpr int StageABytes = BM * BK * 2;
constexpr int threads_of(int epilogue_warps) { return 64 + 32 * epilogue_warps; } // warp 0: TMA, warp 1: MMA, then the epilogue warps
constexpr int ControlBytes = 512;   // barriers, TMEM slot, flags
constexpr int RowScratchBytes = 2 * 4 * BM * 4; // CrossEntropy: row maxima and row sums of the four column shares
constexpr int MaxShared = 232448 - 1024; // 227 KB less the runtime's own reservation
// Where the caller says that others run beside it (GemmArgs::beside_others), a batched product of at most one tile per SM, up to 128
// columns wide, runs in half an SM: eight epilogue warps, one accumulator of its own width, and a ring of half the shared memory.
// Measured with Newton-Schulz products as launches of their own, four chains of them beside each other: of 60 in a step of 6 layers
// d 384 the 45 of 128 columns, 108 blocks each, as whole SMs were kept waiting for one another (eight optimizer steps
// 4.56 -> 3.82 ms, 6 layers d 320 3.92 -> 3.10, the same bits; two blocks to an SM above one tile per SM measured level).  Products in a chain of their own,
// a sharded optimizer's among them, keep the deep ring: tg_predict of 12 layers d 768 takes 838 us with halves, 735 without.  Every kernel that takes tensor memory lets its
// dependents launch only once it holds it, so none can wait for columns that a kernel waiting for it holds.
constexpr int HalfShared = 113 * 1024;

struct TcParams {
    int m, n, k, batch;
    int bn;                 // tile width
    int a_mn, b_mn;         // operand majorness
    int splits, k_blocks_per_split;
    int epilogue, out_fp32;
    int stages;             // depth of the operand ring
    int tmem_columns;
    int wide;               // C, C2 and R rows are 32-byte aligned: 256-bit epilogue accesses
    int reduce_later;       // K splits only write their partial tiles; splitk_reduce_kernel adds them afterwards
    void *c, *c2;
    const void *r;
    long long ldc, ldr, c_batch, r_batch;
    float alpha, beta;
    float *workspace;       // [splits][batch][m_tiles*BM][n_tiles*bn] FP32 partial tiles
    unsigned *tickets;      // one per output tile, zero between launches
    StepCounters *counters;
};

// Two BF16 values of a word as a pair of FP32 ones (the lower half first), and back.
__device__ __forceinline__ uint64_t unpack_pair(uint32_t packed) {
    return float_pair(__uint_as_float(packed << 16), __uint_as_float(packed & 0xffff0000u));
}
__device__ __forceinline__ uint32_t pack_pair(uint64_t v) {
    float lo, hi;
    split_pair(v, lo, hi);
    return pack_bf16(lo, hi);
}
__device__ __forceinline__ uint64_t both(float v) { return float_pair(v, v); }

// gelu(x) = x Phi(x) and gelu'(x) = Phi(x) + x phi(x) of two BF16 values, as BF16.
// Phi(x) = 0.5 (1 + erf(x / sqrt 2)) by Abramowitz & Stegun 7.1.26 (|error| < 3e-7) with every
// constant folded: t = 1 / (1 + p |x| / sqrt 2), e = 2^(-x^2 log2(e) / 2), tail = 0.5 erfc = poly(t) t e.
// Two SFU operations (rcp, ex2) per value; the exponential also gives the Gaussian density of the derivative.  Issue slots bound
// this epilogue: in pairs it takes 14 instructions a value, one value at a time 25.
template <bool Derivative>
__device__ __forceinline__ void gelu_pair(uint32_t packed, uint32_t &activated, uint32_t &derivative) {
    const uint64_t x = unpack_pair(packed), magnitude = unpack_pair(packed & 0x7fff7fffu);
    float d0, d1, q0, q1, t0, t1, e0, e1;
    split_pair(fma_pair(both(0.23164189f), magnitude, both(1.f)), d0, d1);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t0) : "f"(d0));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t1) : "f"(d1));
    split_pair(mul_pair(mul_pair(both(-0.72134752f), x), x), q0, q1);
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(q0));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(q1));
    const uint64_t t = float_pair(t0, t1), e = float_pair(e0, e1);
    uint64_t poly = fma_pair(t, both(0.5307027145f), both(-0.7265760135f));
    poly = fma_pair(t, poly, both(0.7107068705f));
    poly = fma_pair(t, poly, both(-0.142248368f));
    poly = fma_pair(t, poly, both(0.127414796f));
    const uint64_t tail = mul_pair(mul_pair(poly, t), e), rest = fma_pair(tail, both(-1.f), both(1.f));
    float x0, x1, a0, a1, b0, b1;
    split_pair(x, x0, x1);
    split_pair(tail, a0, a1);
    split_pair(rest, b0, b1);
    const uint64_t cdf = float_pair(x0 >= 0.f ? b0 : a0, x1 >= 0.f ? b1 : a1);
    activated = pack_pair(mul_pair(x, cdf));
    if (Derivative)
        derivative = pack_pair(fma_pair(x, mul_pair(both(0.3989422804014327f), e), cdf)); // exp(-x^2/2) / sqrt(2 pi)
}

// Direct global store of eight consecutive outputs (split-K reduction path only).
__device__ __forceinline__ void store_group(const TcParams &p, float (&v)[8], long long row, int col, int z) {
    const long long ci = z * p.c_batch + row * p.ldc + col;
    if (p.out_fp32)
        store8((float *)p.c + ci, v);
    else
        store8((bf16 *)p.c + ci, v);
}

// The epilogue threads meet (named barrier 1), with the AND of a predicate over them.
template <int Warps> __device__ __forceinline__ void epilogue_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(32 * Warps) : "memory"); }
template <int Warps> __device__ __forceinline__ bool epilogue_all(bool ok) {
    uint32_t result;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, 1, %2, p;\n\t"
                 "selp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(result)
                 : "r"(uint32_t(ok)), "n"(32 * Warps)
                 : "memory");
    return result != 0;
}

// Where a work item lies: the K splits of a tile follow one another, tiles run along n first, matrices of a batch last.  In 32 bits
// (see MostItems): 64-bit divisions cost every warp some 500 instructions an item.
struct Item {
    int split, tile, nt, mt, z;
};
__device__ __forceinline__ Item locate(const TcParams &p, int work, int n_tiles, int m_units, int unit, int rank) {
    Item i;
    i.split = 0, i.tile = work, i.z = 0;
    if (p.splits > 1) {
        i.tile = work / p.splits;
        i.split = work - i.tile * p.splits;
    }
    int m = i.tile / n_tiles;
    i.nt = i.tile - m * n_tiles;
    if (p.batch > 1) {
        i.z = m / m_units;
        m -= i.z * m_units;
    }
    i.mt = m * unit + rank;
    return i;
}

// Pair = true: the CTA is half of a cluster of two that computes a 256-row tile with
// cta_group::2 MMAs issued by the pair's first CTA.  Each CTA stages its own 128 rows of A and half
// of the B tile (the tensor core reads the other half from the partner's shared memory), so a
// K block costs each SM 16 KB + BN/2 x 128 B instead of 16 KB + BN x 128 B and the ring is deeper.
template <int Kind, bool OutFp32, bool Pair, int EpilogueWarps, bool EarlyB = false>
__global__ void __launch_bounds__(threads_of(EpilogueWarps), EpilogueWarps == 8 ? 2 : 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, TcParams p) {
    extern __shared__ uint8_t raw_shared[];
    const uint32_t base = (smem_address(raw_shared) + 1023u) & ~1023u;
    uint8_t *aligned = raw_shared + (base - smem_address(raw_shared));
    constexpr int Unit = Pair ? 2 : 1;
    const uint32_t rank = Pair ? cluster_rank() : 0u;
    const int bn_local = p.bn / Unit; // B rows staged by this CTA
    const int stage_bytes = StageABytes + bn_local * BK * 2;
    uint64_t *barriers = reinterpret_cast<uint64_t *>(aligned + p.stages * stage_bytes);
    // barriers: full[8], empty[8], tmem_full[2], tmem_empty[2]
    const uint32_t full0 = smem_address(barriers), empty0 = full0 + 8 * MaxStages, tfull0 = empty0 + 8 * MaxStages,
                   tempty0 = tfull0 + 16;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(barriers + 2 * MaxStages + 4);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    volatile int *last_split_flag = reinterpret_cast<volatile int *>(tmem_slot + 2);

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbarrier_init(full0 + 8 * s, 1);
            mbarrier_init(empty0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbarrier_init(tfull0 + 8 * b, 1);
            mbarrier_init(tempty0 + 8 * b, EpilogueWarps * Unit);
        }
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_map(&map_a);
        prefetch_map(&map_b);
    }
    if (warp == 1) {
        if constexpr (Pair) {
            tmem_alloc_pair(smem_address(tmem_slot), p.tmem_columns);
            tmem_relinquish_pair();
        } else {
            tmem_alloc(smem_address(tmem_slot), p.tmem_columns);
            tmem_relinquish();
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if constexpr (Pair)
        cluster_sync_all(); // the partner's barriers exist before anything signals them
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // Barriers, tensor memory and descriptors are set up; only now wait for the kernel before this one
    // (its tail overlaps the set-up above when this kernel was launched programmatically).
    grid_launch_dependents();
    if (!EarlyB || warp != 0)
        grid_dependency_wait();

    // Tiles along M are scheduled per CTA pair; m_tiles counts 128-row tiles including padding.
    const int m_tiles = ((p.m + BM * Unit - 1) / (BM * Unit)) * Unit, n_tiles = (p.n + p.bn - 1) / p.bn;
    const int k_blocks = (p.k + BK - 1) / BK;
    const int m_units = m_tiles / Unit;
    const int work_items = m_units * n_tiles * p.batch * p.splits;
    const int first_item = int(blockIdx.x) / Unit, item_stride = int(gridDim.x) / Unit;
    const uint32_t stage_tx = stage_bytes * Unit; // bytes landing for one stage in both CTAs

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (elect_one()) {
            // Both CTAs' bytes are counted on the first CTA's barrier, armed by that CTA.
            const uint32_t landed0 = Pair ? cluster_address(full0, 0) : full0;
            // A K-major operand comes as one box of 64 K-elements, an MN-major one as boxes of 64 rows of the tile.
            const int a_dx = p.a_mn ? 0 : BK, a_dy = p.a_mn ? BK : 0, b_dx = p.b_mn ? 0 : BK, b_dy = p.b_mn ? BK : 0;
            const int b_boxes = p.b_mn ? bn_local / 64 : 1;
            int stage = 0;
            uint32_t phase = 0;
            auto load = [&](uint32_t dst, const CUtensorMap *map, int x, int y, int z, uint32_t bar) {
                if constexpr (Pair)
                    tma_load_3d_pair(dst, map, x, y, z, bar);
                else
                    tma_load_3d(dst, map, x, y, z, bar);
            };
            // A weight is there before the activations that it multiplies: the ring's first round of it is fetched while the kernel before this one ends.
            int early = 0; // K blocks whose B is on its way
            if constexpr (EarlyB) {
                if (first_item < work_items) {
                    const Item item = locate(p, first_item, n_tiles, m_units, Unit, int(rank));
                    const int n_first = item.nt * p.bn + int(rank) * bn_local;
                    int bx = p.b_mn ? n_first : 0, by = p.b_mn ? 0 : n_first;
                    for (const int most = min(p.stages, k_blocks); early < most; ++early) {
                        const uint32_t sb = base + early * stage_bytes + StageABytes, bar = landed0 + 8 * early;
                        if (rank == 0)
                            mbarrier_expect_tx(full0 + 8 * early, stage_tx);
                        for (int j = 0; j < b_boxes; ++j)
                            load(sb + j * 64 * BK * 2, &map_b, bx + j * 64, by, item.z, bar);
                        bx += b_dx, by += b_dy;
                    }
                }
                grid_dependency_wait();
            }
            for (int w = first_item; w < work_items; w += item_stride) {
                const Item item = locate(p, w, n_tiles, m_units, Unit, int(rank));
                const int kb0 = item.split * p.k_blocks_per_split;
                const int kb1 = min(k_blocks, kb0 + p.k_blocks_per_split);
                const int m_first = item.mt * BM, n_first = item.nt * p.bn + int(rank) * bn_local, z = item.z;
                int ax = p.a_mn ? m_first : kb0 * BK, ay = p.a_mn ? kb0 * BK : m_first;
                int bx = p.b_mn ? n_first : kb0 * BK, by = p.b_mn ? kb0 * BK : n_first;
                bool ok = true;
                int kb = kb0;
                if constexpr (EarlyB) {
                    for (; early; --early, ++kb) { // nothing has used these stages yet
                        const uint32_t sa = base + stage * stage_bytes, bar = landed0 + 8 * stage;
                        load(sa, &map_a, ax, ay, z, bar);
                        if (p.a_mn)
                            load(sa + 64 * BK * 2, &map_a, ax + 64, ay, z, bar);
                        ax += a_dx, ay += a_dy, bx += b_dx, by += b_dy;
                        if (++stage == p.stages) {
                            stage = 0;
                            phase ^= 1;
                        }
                    }
                }
                for (; kb < kb1; ++kb) {
                    ok = mbarrier_wait(empty0 + 8 * stage, phase ^ 1, abort_flag, p.counters, 101);
                    if (!ok)
                        break;
                    const uint32_t sa = base + stage * stage_bytes, sb = sa + StageABytes, bar = landed0 + 8 * stage;
                    if (rank == 0)
                        mbarrier_expect_tx(full0 + 8 * stage, stage_tx);
                    load(sa, &map_a, ax, ay, z, bar);
                    if (p.a_mn)
                        load(sa + 64 * BK * 2, &map_a, ax + 64, ay, z, bar);
                    load(sb, &map_b, bx, by, z, bar);
                    for (int j = 1; j < b_boxes; ++j)
                        load(sb + j * 64 * BK * 2, &map_b, bx + j * 64, by, z, bar);
                    ax += a_dx, ay += a_dy, bx += b_dx, by += b_dy;
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
        // ---------------- MMA issuer ----------------
        if (rank == 0 && elect_one()) {
            const uint32_t instruction = instruction_descriptor(BM * Unit, p.bn, p.a_mn, p.b_mn);
            // Per 16-element K step inside a stage: 32 bytes along a K-major row, or 16 rows of
            // 128 bytes for an MN-major operand.
            const uint32_t a_step = p.a_mn ? 16 * 128 : 32, b_step = p.b_mn ? 16 * 128 : 32;
            // the first stage's descriptors; the products only move them along
            const uint64_t a_desc = smem_descriptor(base, p.a_mn ? 64 * BK * 2 : 16, 1024),
                           b_desc = smem_descriptor(base + StageABytes, p.b_mn ? 64 * BK * 2 : 16, 1024);
            auto commit = [](uint32_t bar) { // arrives once the products issued so far are done, in both CTAs of a pair
                if constexpr (Pair)
                    tcgen05_commit_both(bar);
                else
                    tcgen05_commit(bar);
            };
            int stage = 0, buffer = 0;
            uint32_t phase = 0, buffer_phase = 0;
            for (int w = first_item; w < work_items; w += item_stride) {
                const int kb0 = p.splits > 1 ? w % p.splits * p.k_blocks_per_split : 0;
                const int kb1 = min(k_blocks, kb0 + p.k_blocks_per_split);
                if (!mbarrier_wait(tempty0 + 8 * buffer, buffer_phase ^ 1, abort_flag, p.counters, 102))
                    break;
                tcgen05_fence_after();
                const uint32_t accumulator = tmem_base + buffer * MaxBN;
                bool ok = true;
                for (int kb = kb0; kb < kb1; ++kb) {
                    ok = mbarrier_wait(full0 + 8 * stage, phase, abort_flag, p.counters, 103);
                    if (!ok)
                        break;
                    tcgen05_fence_after();
                    const uint64_t da = descriptor_at(a_desc, stage * stage_bytes), db = descriptor_at(b_desc, stage * stage_bytes);
#pragma unroll
                    for (int ks = 0; ks < BK / 16; ++ks) {
                        const uint64_t dak = descriptor_at(da, ks * a_step), dbk = descriptor_at(db, ks * b_step);
                        if constexpr (Pair)
                            tcgen05_mma_bf16_pair(accumulator, dak, dbk, instruction, (kb > kb0 || ks > 0) ? 1u : 0u);
                        else
                            tcgen05_mma_bf16(accumulator, dak, dbk, instruction, (kb > kb0 || ks > 0) ? 1u : 0u);
                    }
                    commit(empty0 + 8 * stage); // frees the stage once these products have read it
                    if (++stage == p.stages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (!ok)
                    break;
                commit(tfull0 + 8 * buffer); // the accumulator is complete
                if (++buffer == 2) {
                    buffer = 0;
                    buffer_phase ^= 1;
                }
            }
        }
    } else {
        // ---------------- epilogue: 16 (8) warps; warps q, q+4, .. share TMEM lanes 32q..32q+31 and
        // take every fourth (second) 32-column chunk.  Four warps per scheduler hide one another's TMEM,
        // ALU, SFU and global-load latencies (the epilogue math is a dependent chain per element).
        constexpr int Shares = EpilogueWarps / 4;
        const int quarter = warp % 4, share = (warp - 2) / 4;
        constexpr bool has_r = Kind == int(Epilogue::Residual) || Kind == int(Epilogue::GeluGrad) ||
                               Kind == int(Epilogue::Axpby);
        constexpr bool whole_rows = Kind == int(Epilogue::CrossEntropy); // the sixteen warps meet per tile
        // A lane drains its own row of tensor memory, and stores (and reads of the second tensor) half of its own and half of its
        // neighbour's: see exchange_rows.
        const bool odd = lane & 1;
        auto row_of = [&](const Item &item) { return (long long)item.mt * BM + quarter * 32 + (lane & ~1); }; // the pair's first row
        auto fetch_second = [&](const Item &item, int c, uint32_t (&rv)[2][8]) { // the second tensor's part of a chunk
            const int column = item.nt * p.bn + c * 32 + (odd ? 16 : 0);
            const long long row = row_of(item);
            if (!has_r || column >= p.n)
                return;
            const bf16 *src = (const bf16 *)p.r + item.z * p.r_batch + row * p.ldr + column;
#pragma unroll
            for (int g = 0; g < 2; ++g)
                if (row + g < p.m)
                    load_global32(src + g * p.ldr, rv[g], p.wide && column + 16 <= p.n, column + 8 < p.n);
        };
        // The second tensor's chunk is fetched one chunk ahead, over the end of a tile too: where products are short the
        // accumulators are ready before the epilogue gets to them, and nothing else would hide these loads.
        uint32_t rv[2][8];
        auto item_of = [&](int w) { return locate(p, w, n_tiles, m_units, Unit, int(rank)); };
        if (has_r && first_item < work_items && share * 32 < p.bn)
            fetch_second(item_of(first_item), share, rv);
        int buffer = 0;
        uint32_t buffer_phase = 0;
        for (int w = first_item; w < work_items; w += item_stride) {
            const Item item = item_of(w);
            const int nt = item.nt, mt = item.mt, z = item.z, split = item.split;
            bool ready = mbarrier_wait(tfull0 + 8 * buffer, buffer_phase, abort_flag, p.counters, 104);
            if (p.splits > 1 || whole_rows) // the warps meet at named barriers below: leave together or not at all
                ready = epilogue_all<EpilogueWarps>(ready);
            if (!ready)
                break;
            tcgen05_fence_after();
            const uint32_t taddr = tmem_base + (uint32_t(quarter * 32) << 16) + buffer * MaxBN;
            const int tile_columns = min(p.bn, p.n - nt * p.bn);
            const int chunks = (tile_columns + 31) / 32;
            auto release = [&] { // the accumulator has been read: the products of the tile after the next may overwrite it
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if constexpr (Pair)
                        mbarrier_arrive_cluster(cluster_address(tempty0 + 8 * buffer, 0));
                    else
                        mbarrier_arrive(tempty0 + 8 * buffer);
                }
            };
            if constexpr (whole_rows) {
                // One 256-column tile holds whole rows of logits.  A thread owns row `row` in the 32-column chunks
                // `share` and `share + 4`; the four shares of a row exchange their maxima and sums through shared
                // memory and add them in share order.
                float *row_high = reinterpret_cast<float *>(aligned + p.stages * stage_bytes + ControlBytes);
                float *row_sum = row_high + Shares * BM;
                const int local = quarter * 32 + lane;
                const long long row = (long long)mt * BM + local;
                const int target = row < p.m ? static_cast<const uint8_t *>(p.r)[row] : 0;
                // Three passes over the thread's 64 columns, 16 at a time; the exponentials replace the logits in tensor memory.  With
                // the 64 columns in registers the epilogue of a tile took 16000 clocks (unrolled code that runs once, and 250 bytes
                // of spills), like this 8900.
                auto first_column = [&](int piece) { return (share + piece / 2 * Shares) * 32 + piece % 2 * 16; };
                float high = -CUDART_INF_F, picked = 0.f;
#pragma unroll 1
                for (int piece = 0; piece < 4; ++piece) {
                    uint32_t v[16];
                    tmem_load_32x16_async(taddr + first_column(piece), v);
                    const int at = target - first_column(piece);
                    tmem_wait_load(v);
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        high = fmaxf(high, __uint_as_float(v[j]));
                        picked = j == at ? __uint_as_float(v[j]) : picked;
                    }
                }
                row_high[share * BM + local] = high;
                epilogue_barrier<EpilogueWarps>();
                high = fmaxf(fmaxf(row_high[local], row_high[BM + local]), fmaxf(row_high[2 * BM + local], row_high[3 * BM + local]));
                float sum = 0.f;
#pragma unroll 1
                for (int piece = 0; piece < 4; ++piece) {
                    uint32_t v[16];
                    tmem_load_32x16_async(taddr + first_column(piece), v);
                    tmem_wait_load(v);
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float e = expf(__uint_as_float(v[j]) - high);
                        sum += e;
                        v[j] = __float_as_uint(e);
                    }
                    tmem_store_32x16(taddr + first_column(piece), v);
                }
                tmem_wait_store();
                row_sum[share * BM + local] = sum;
                epilogue_barrier<EpilogueWarps>();
                sum = ((row_sum[local] + row_sum[BM + local]) + row_sum[2 * BM + local]) + row_sum[3 * BM + local];
                if (row < p.m && target / 32 % Shares == share)
                    static_cast<float *>(p.c2)[row] = high + logf(sum) - picked;
                if (p.c) {
                    const float inverse = 1.f / sum;
#pragma unroll 1
                    for (int half = 0; half < 2; ++half) {
                        uint32_t out[16];
#pragma unroll
                        for (int g = 0; g < 2; ++g) {
                            const int column = first_column(half * 2 + g), at = target - column;
                            uint32_t v[16];
                            tmem_load_32x16_async(taddr + column, v);
                            tmem_wait_load(v);
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                const float a = (__uint_as_float(v[2 * j]) * inverse - (2 * j == at ? 1.f : 0.f)) * p.alpha;
                                const float b = (__uint_as_float(v[2 * j + 1]) * inverse - (2 * j + 1 == at ? 1.f : 0.f)) * p.alpha;
                                out[g * 8 + j] = pack_bf16(a, b);
                            }
                        }
                        exchange_rows(out, out + 8, odd);
                        const long long row0 = row_of(item);
                        bf16 *dst = (bf16 *)p.c + row0 * p.ldc + first_column(half * 2) + (odd ? 16 : 0);
#pragma unroll
                        for (int g = 0; g < 2; ++g)
                            if (row0 + g < p.m)
                                store_global32(dst + g * p.ldc, out + g * 8, p.wide, true);
                    }
                }
                release();
            } else if (Kind != int(Epilogue::Store) || p.splits == 1) {
                const long long row = row_of(item), c_row = z * p.c_batch + row * p.ldc;
                for (int c = share; c < chunks; c += Shares) {
                    const bool last = c + Shares >= chunks;
                    const int chunk_column = nt * p.bn + c * 32;
                    if constexpr (OutFp32) {
                        uint32_t acc[32];
                        tmem_load_32x32_async(taddr + c * 32, acc);
                        tmem_wait_load(acc);
                        if (last)
                            release();
#pragma unroll
                        for (int half = 0; half < 2; ++half) {
                            exchange_rows(acc + half * 16, acc + half * 16 + 8, odd);
                            const int column = chunk_column + half * 16 + (odd ? 8 : 0);
#pragma unroll
                            for (int g = 0; g < 2; ++g)
                                if (row + g < p.m && column < p.n)
                                    store_global32((float *)p.c + c_row + g * p.ldc + column, acc + half * 16 + g * 8, p.wide, true);
                        }
                    } else {
                        // the chunk's row as BF16: sums of the products, for Axpby the results
                        uint32_t v[16], ahead[2][8];
                        if constexpr (has_r) {
                            if constexpr (Kind == int(Epilogue::Axpby))
                                exchange_rows(rv[0], rv[1], odd); // to lane = row
#pragma unroll
                            for (int half = 0; half < 2; ++half) { // 16 columns at a time: 32, and twice the second tensor, would spill
                                uint32_t acc[16];
                                tmem_load_32x16_async(taddr + c * 32 + half * 16, acc);
                                if (half == 0) {
                                    if (!last)
                                        fetch_second(item, c + Shares, ahead);
                                    else if (w + item_stride < work_items)
                                        fetch_second(item_of(w + item_stride), share, ahead);
                                }
                                tmem_wait_load(acc);
#pragma unroll
                                for (int j = 0; j < 8; ++j) {
                                    const float s0 = __uint_as_float(acc[2 * j]), s1 = __uint_as_float(acc[2 * j + 1]);
                                    if constexpr (Kind == int(Epilogue::Axpby))
                                        v[half * 8 + j] = pack_bf16(p.alpha * s0 + p.beta * __uint_as_float(rv[half][j] << 16),
                                                                    p.alpha * s1 + p.beta * __uint_as_float(rv[half][j] & 0xffff0000u));
                                    else
                                        v[half * 8 + j] = pack_bf16(s0, s1);
                                }
                            }
                        } else {
                            uint32_t acc[32];
                            tmem_load_32x32_async(taddr + c * 32, acc);
                            tmem_wait_load(acc);
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                v[j] = pack_bf16(__uint_as_float(acc[2 * j]), __uint_as_float(acc[2 * j + 1]));
                        }
                        if (last)
                            release();
                        exchange_rows(v, v + 8, odd);
                        const int column = chunk_column + (odd ? 16 : 0);
                        const bool whole = p.wide && column + 16 <= p.n, second = column + 8 < p.n;
#pragma unroll
                        for (int g = 0; g < 2; ++g) {
                            uint32_t out[8], activated[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j) { // two columns at a time
                                const uint32_t sum = v[g * 8 + j];
                                if constexpr (Kind == int(Epilogue::Residual))
                                    out[j] = pack_pair(add_pair(unpack_pair(sum), unpack_pair(rv[g][j])));
                                else if constexpr (Kind == int(Epilogue::GeluGrad))
                                    out[j] = pack_pair(mul_pair(unpack_pair(sum), unpack_pair(rv[g][j])));
                                else if constexpr (Kind == int(Epilogue::GeluDual))
                                    gelu_pair<true>(sum, activated[j], out[j]); // out: gelu'(pre)
                                else if constexpr (Kind == int(Epilogue::Gelu))
                                    gelu_pair<false>(sum, out[j], activated[j]);
                                else
                                    out[j] = sum;
                            }
                            if (row + g < p.m && column < p.n) {
                                const long long at = c_row + g * p.ldc + column;
                                store_global32((bf16 *)p.c + at, out, whole, second);
                                if constexpr (Kind == int(Epilogue::GeluDual))
                                    store_global32((bf16 *)p.c2 + at, activated, whole, second);
                            }
                        }
                        if constexpr (has_r) {
#pragma unroll
                            for (int g = 0; g < 2; ++g)
#pragma unroll
                                for (int j = 0; j < 8; ++j)
                                    rv[g][j] = ahead[g][j];
                        }
                    }
                }
                if (share >= chunks) { // no chunk of this tile, perhaps one of the next
                    release();
                    if (has_r && w + item_stride < work_items && share * 32 < p.bn)
                        fetch_second(item_of(w + item_stride), share, rv);
                }
            } else {
                // Partial tile to the workspace (padded to whole tiles, so no bounds checks).  A 32 x 32
                // chunk is stored column by column (lane = row), so every access is one 128-byte line.
                const long long padded_m = (long long)m_tiles * BM, padded_n = (long long)n_tiles * p.bn;
                const long long split_stride = (long long)p.batch * padded_m * padded_n;
                float *partial = p.workspace + ((long long)split * p.batch + z) * padded_m * padded_n;
                const long long chunk_row = ((long long)mt * 4 + quarter) * (padded_n / 32) + nt * (p.bn / 32);
                for (int chunk = share; chunk < p.bn / 32; chunk += Shares) {
                    float v[32];
                    tmem_load_32x32(taddr + chunk * 32, v);
                    float *out = partial + (chunk_row + chunk) * 1024 + lane;
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        out[j * 32] = v[j];
                }
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if constexpr (Pair)
                        mbarrier_arrive_cluster(cluster_address(tempty0 + 8 * buffer, 0));
                    else
                        mbarrier_arrive(tempty0 + 8 * buffer);
                }
                if (p.reduce_later) { // many splits: one SM adding them all would take longer than the products
                    if (++buffer == 2) {
                        buffer = 0;
                        buffer_phase ^= 1;
                    }
                    continue;
                }
                // Ticket: the split that arrives last reduces the tile in split order.
                __threadfence();
                epilogue_barrier<EpilogueWarps>();
                if (threadIdx.x == 64) {
                    unsigned ticket = atomicAdd(&p.tickets[item.tile * Unit + rank], 1u);
                    int last = ticket == unsigned(p.splits - 1);
                    if (last)
                        p.tickets[item.tile * Unit + rank] = 0; // ready for the next launch
                    last_split_flag[0] = last;
                }
                epilogue_barrier<EpilogueWarps>();
                if (last_split_flag[0]) {
                    const long long row = (long long)mt * BM + quarter * 32 + lane;
                    __threadfence();
                    for (int chunk = share; chunk < p.bn / 32; chunk += Shares) {
                        const int column = nt * p.bn + chunk * 32;
                        if (column >= p.n)
                            break;
                        // L2 only (__ldcg): the partials were written by other SMs.
                        const float *src = p.workspace + ((long long)z * padded_m * padded_n) +
                                           (chunk_row + chunk) * 1024 + lane;
                        float sum[32];
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            sum[j] = 0.f;
                        for (int sp = 0; sp < p.splits; ++sp) {
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                sum[j] += __ldcg(src + sp * split_stride + j * 32);
                        }
                        if (row < p.m) {
#pragma unroll
                            for (int g = 0; g < 4; ++g) {
                                if (column + g * 8 >= p.n)
                                    break;
                                float group[8];
#pragma unroll
                                for (int j = 0; j < 8; ++j)
                                    group[j] = sum[g * 8 + j];
                                store_group(p, group, row, column + g * 8, z);
                            }
                        }
                    }
                }
                epilogue_barrier<EpilogueWarps>(); // last_split_flag is reused next tile
            }
            if (++buffer == 2) {
                buffer = 0;
                buffer_phase ^= 1;
            }
        }
    }

    // Teardown.  After an aborted wait, give copies already in flight time to land before the
    // shared memory and tensor memory are released.
    __syncthreads();
    if (*abort_flag)
        __nanosleep(2000000);
    tcgen05_fence_before();
    __syncthreads();
    if constexpr (Pair) {
        cluster_sync_all(); // neither CTA's tensor or shared memory is released while the other may touch it
        if (warp == 1)
            tmem_dealloc_pair(tmem_base, p.tmem_columns);
    } else {
        if (warp == 1)
            tmem_dealloc(tmem_base, p.tmem_columns);
    }
}

// C = the K splits' partial tiles added in split order, for schedules with four or more splits: there the last
// arriver of a tile would pull every partial tile through one SM (1 MB per CTA at eight splits: 24 000 clocks,
// as long as the products themselves); this kernel spreads the same additions, in the
// same order, over the whole GPU.  One block per 32 x 32 chunk of the padded output (a chunk is stored column
// by column, see the kernel above); rows go out whole through a padded shared-memory tile.
template <bool OutFp32>
__global__ void __launch_bounds__(256) splitk_reduce_kernel(TcParams p, long long padded_m, long long padded_n) {
    __shared__ float tile[32][33];
    const long long chunks_per_row = padded_n / 32, chunks_per_matrix = (padded_m / 32) * chunks_per_row;
    const long long chunk = blockIdx.x % chunks_per_matrix;
    const int z = int(blockIdx.x / chunks_per_matrix);
    const long long split_stride = (long long)p.batch * padded_m * padded_n;
    const float *source = p.workspace + (long long)z * padded_m * padded_n + chunk * 1024;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int e = threadIdx.x + 256 * u; // column e / 32, row e % 32 of the chunk
        float sum = 0.f;
        for (int split = 0; split < p.splits; ++split)
            sum += __ldcg(source + split * split_stride + e);
        tile[e / 32][e % 32] = sum;
    }
    __syncthreads();
    const long long row = chunk / chunks_per_row * 32 + threadIdx.x / 8;
    const int column = int(chunk % chunks_per_row) * 32 + (threadIdx.x % 8) * 4;
    if (row >= p.m || column >= p.n)
        return;
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        v[i] = tile[(threadIdx.x % 8) * 4 + i][threadIdx.x / 8];
    const long long index = z * p.c_batch + row * p.ldc + column;
    if (column + 4 <= p.n && p.wide) {
        if constexpr (OutFp32)
            *reinterpret_cast<float4 *>((float *)p.c + index) = make_float4(v[0], v[1], v[2], v[3]);
        else
            *reinterpret_cast<uint2 *>((bf16 *)p.c + index) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
    } else {
        for (int i = 0; i < 4 && column + i < p.n; ++i) {
            if constexpr (OutFp32)
                ((float *)p.c)[index + i] = v[i];
            else
                ((bf16 *)p.c)[index + i] = __float2bfloat16(v[i]);
        }
    }
}

// ---------------------------------------------------------------------------- host side ------
struct Schedule {
    int bn = 0, splits = 1, k_blocks_per_split = 0, pair = 0;
};

// What a schedule costs, in nanoseconds: launch + rounds of tiles x (64-deep K blocks x block + tile).  Fitted to 832 products
// of 256 to 32768 tokens and widths 128 to 1024 (activations and input gradients, K-major and MN-major B), each timed with every
// tile width, single and paired; the model reproduces the times within 5 to 8 % and its choice is 0.3 % slower than the best of
// each (geometric mean).  The costs below for rows off the cache lines are fitted to 824 more, of odd multiples of eight: without
// them the choice was 1.6 % slower than the best of each and in the worst cases took wide single tiles where pairs of them, which
// stage fewer lines, were a third faster; with them 0.9 %.  A pair's launch costs 0.9 us more and its tiles take longer to hand over, single CTAs read more
// operand bytes per product: pairs are for many rounds over a long K.  The model before it (MMA and shared-memory clocks, no
// launch or tile times) chose 8 % slower on average: 4096 x 768 x 2304 17.4 -> 13.9 us, 8192 x 2048 x 512 25.1 -> 18.5,
// 1024 x 2304 x 768 7.5 -> 6.4, 32768 x 512 x 128 21.9 -> 13.5.  The tile's shape does not change a result: every element
// adds its products in ascending k.
struct TileCost {
    int bn, block, tile;
};
constexpr TileCost SingleCost[] = {{256, 342, 1500}, {192, 262, 1280}, {128, 209, 940}, {64, 184, 550}};
constexpr TileCost PairCost[] = {{256, 284, 2100}, {192, 211, 1900}, {128, 188, 1450}};
constexpr int SingleLaunch = 3240, PairLaunch = 4100;
// Rows that do not start on a cache line take two of them for one, and those off a 32-byte sector five sectors for four: picoseconds
// per 128-byte line of an operand and 64-deep K block (the first is hidden where a pair stages half of B).  Rows of C off a sector
// are written in parts: nanoseconds per tile column.
constexpr int LineCost = 140, SectorCost = 500, RaggedStoreCost = 4;
// Where N is whole 64-column blocks, as a model's are: costs fitted to 2698 products of 512 to 40000 tokens and models of widths 128 to 1024
// (K and N up to 4096, one of them at most 1024), in every form.  A pair's tile costs half of what it did when its warps awaited their stores
// before they handed an accumulator over.  The choice is 1.0 % slower than the best form (a third of the products kept out of the fit); by the costs above
// 3.0 %.  Over 19853 others of 256 to 65536 tokens, N and K of 128 to 4096, it is 0.5 % slower than the best form (0.5 % over K up to 1024, 0.4 up to
// 2048, 0.7 above; at worst 38 %), by the costs above 2.4 %, and over 6916 with K off whole blocks 0.4 and 1.8.
// 32768 x 768 x 768 41.0 -> 34.6 us, 8192 x 3072 x 768 32.2 -> 27.6, 4096 x 3072 x 768 18.0 -> 15.9.  How often K is cut stays with the costs above: it
// decides the order of the sums.
constexpr TileCost WholeSingleCost[] = {{256, 312, 1090}, {192, 259, 999}, {128, 199, 633}, {64, 142, 391}};
constexpr TileCost WholePairCost[] = {{256, 305, 725}, {192, 227, 781}, {128, 179, 494}};
constexpr int WholeSingleLaunch = 2890, WholePairLaunch = 3719;
// They know nothing of where A comes from.  Where it does not stay in L2, its 128 rows of a stage are what a CTA waits for, and the ring of
// a 256-column single tile holds four of them to a pair's six: from 64 MB of A on, where the costs take that tile, the pair is 1.5 % faster up
// to 80 MB and 6.6 % above (27 products; 17871 x 256 x 3456 36.6 and 30.4 us), up to 48 MB it is 3 % slower (1273).
constexpr int64_t StreamedBytes = int64_t(64) << 20;
// A K split of n: partial tiles, fence, ticket and read-back by one SM, or from four on a second launch, and the partial tiles'
// passes through memory.
constexpr long long split_cost(int splits, int bn, long long outputs) {
    return splits == 1 ? 0 : 4500 + (splits < 4 ? 20 * bn : 0) + splits * outputs / 1000;
}
Schedule product_schedule(const GemmArgs &g, int sms) {
    const bool b_mn = g.b_col != 1;
    const bool plain = g.epilogue == Epilogue::Store; // K is split only for plain stores
    const bool whole_rows = g.epilogue == Epilogue::CrossEntropy; // a tile must hold complete rows
    const int m_tiles = (g.m + BM - 1) / BM, k_blocks = (g.k + BK - 1) / BK;
    const int64_t a_pitch = g.a_col == 1 ? g.a_row : g.a_col, b_pitch = b_mn ? g.b_col : g.b_row; // elements of two bytes
    auto lines_off = [&](int bytes, int b_rows) { return (a_pitch * 2 % bytes ? BM : 0) + (b_pitch * 2 % bytes ? b_rows : 0); };
    Schedule best;
    long long best_time = 0;
    // `splits_allowed`: 0 for any number of them, at the costs of aligned rows; otherwise that many, at the operands' own costs.
    auto consider = [&](const TileCost &cost, int unit, int launch, int splits_allowed) {
        const int bn = cost.bn, slots = sms / unit;
        if ((bn > 64 && bn - 64 >= g.n) || (whole_rows && bn != 256))
            return; // a narrower tile already covers N
        if (unit == 2 && b_mn && bn == 192)
            return; // each CTA stages bn/2 rows of B: whole 64-row blocks when B is MN-major
        int block = cost.block, tile = cost.tile;
        if (splits_allowed) {
            block += ((unit == 1 ? LineCost * lines_off(128, bn) : 0) + SectorCost * lines_off(32, bn / unit)) / 1000;
            tile += g.ldc * int(dtype_size(g.out)) % 32 ? RaggedStoreCost * bn : 0;
        }
        const long long tiles = (long long)((m_tiles + unit - 1) / unit) * ((g.n + bn - 1) / bn) * g.batch;
        for (int splits : {1, 2, 3, 4, 6, 8, 12, 16}) {
            const int per = (k_blocks + splits - 1) / splits;
            if (splits > 1 && (!plain || k_blocks / splits < 8 || tiles * splits > slots || (k_blocks + per - 1) / per != splits))
                continue; // the last: would leave an empty split
            if (splits_allowed && splits != splits_allowed)
                continue;
            const long long rounds = (tiles * splits + slots - 1) / slots;
            const long long time = launch + rounds * ((long long)per * block + tile) + split_cost(splits, bn, (long long)g.m * g.n * g.batch);
            if (!best.bn || time < best_time)
                best.bn = bn, best.splits = splits, best.k_blocks_per_split = per, best.pair = unit == 2, best_time = time;
        }
    };
    auto consider_all = [&](int splits_allowed) {
        const bool whole = splits_allowed == 1 && g.n % 64 == 0 && g.batch == 1, streamed = whole && int64_t(g.m) * g.k * 2 > StreamedBytes;
        best = {};
        if (m_tiles >= 2 && sms >= 2)
            for (const TileCost &cost : whole ? WholePairCost : PairCost)
                consider(cost, 2, whole ? WholePairLaunch : PairLaunch, splits_allowed);
        for (const TileCost &cost : whole ? WholeSingleCost : SingleCost)
            if (!(streamed && best.bn && cost.bn == 256))
                consider(cost, 1, whole ? WholeSingleLaunch : SingleLaunch, splits_allowed);
    };
    consider_all(0); // how often K is cut decides the order of the sums: the alignment of the rows has no say in it
    consider_all(best.splits);
    return best;
}

// Weight gradients: FP32 outputs over a long K.  Their schedules were measured in steps rather than alone, where they run beside
// the chain of input gradients: fewer blocks of longer life leave the chain more of the GPU.
// Tile width, K splits and single CTA / CTA pair by a cost model in clocks per 16 of a 64-deep K
// block: the MMA takes bn/2, the shared-memory operand reads (128+bn)/4; a tile adds a fixed drain
// cost and every split one pass over the FP32 partial tile.  CTA pairs (256-row tiles) are tried
// first: they halve the B bytes each SM stages per K block.
// SplitCost, in the model's units (four clocks each: 2000 are about 4.3 us): writing partial tiles, the fence, the
// ticket and reading them back, or a second launch, take 4 to 5 us however small the tiles: 2048 x 256 x 1024 took 12.2 us
// with K cut in two, 8.5 us uncut.  Steps without the cost, with 1000, 2000 and 4000: 4 layers d 256, 2048 tokens 508, 494,
// 455, 454 us; 6 layers d 384, 2331 tokens 1.46, 1.32, 1.22, 1.21 ms; 8 layers d 640, 4096 tokens 2.44, 2.33, 2.28, 2.25 ms.
// (Alone, a weight gradient over 2048 tokens is faster cut in four, 768 x 256 10.4 us against 12.1; beside the chain of
// input gradients the four times as many blocks are in its way: such cuts made the first of these steps 9 % longer.)
// Near-ties are cut: over long K whole schedules, of narrower tiles, take 2 to 5 % longer than the model says.  Whole
// and cut, of 964 shapes the three that this decides: dW 3072 x 768 over 16384 tokens 65.5 and 63.5 us, 768 x 3072 74.1
// and 70.5, 2560 x 640 61.2 and 57.5; at 12000 tokens whole is faster (49.0 and 50.7) and stays, at 32768 the cut by itself.
constexpr int SplitCost = 2000, CutWeight = 48, WholeWeight = 49;
Schedule weight_gradient_schedule(const GemmArgs &g, int sms) {
    const bool b_mn = g.b_col != 1;
    const int m_tiles = (g.m + BM - 1) / BM, k_blocks = (g.k + BK - 1) / BK;
    Schedule best;
    long long best_time = 0;
    for (int unit : {2, 1}) {
        if (unit == 2 && (m_tiles < 2 || sms < 2))
            continue;
        const int slots = sms / unit;
        const long long m_units = (m_tiles + unit - 1) / unit;
        for (int bn : {256, 192, 128, 64}) {
            if (bn > 64 && bn - 64 >= g.n)
                continue; // a narrower tile already covers N
            if (unit == 2 && (bn == 64 || (b_mn && bn == 192)))
                continue; // each CTA stages bn/2 rows of B: whole 64-row blocks when B is MN-major
            const long long tiles = m_units * ((g.n + bn - 1) / bn) * g.batch;
            // Clocks per K block and CTA: the MMA takes bn/2; a single CTA cannot keep its ring full
            // (measured ~65 % of that rate), a pair can.
            const int mma = bn / 2 > (128 + bn) / 4 ? bn / 2 : (128 + bn) / 4;
            const int block_cost = unit == 2 ? mma + 16 : mma * (k_blocks >= 64 ? 9 : 11) / 8 + 16;
            for (int splits : {1, 2, 3, 4, 6, 8, 12, 16}) {
                if (splits > 1 && (k_blocks / splits < 8 || tiles * splits > slots))
                    continue;
                const int per = (k_blocks + splits - 1) / splits;
                if (splits > 1 && (k_blocks + per - 1) / per != splits)
                    continue; // would leave an empty split
                const long long rounds = (tiles * splits + slots - 1) / slots;
                const long long time = splits > 1 ? rounds * ((long long)per * block_cost + bn + splits * bn / 2 + SplitCost) * CutWeight
                                                  : rounds * ((long long)per * block_cost + bn) * WholeWeight;
                if (!best.bn || time < best_time)
                    best.bn = bn, best.splits = splits, best.k_blocks_per_split = per, best.pair = unit == 2,
                    best_time = time;
            }
        }
    }
    return best;
}
Schedule choose_schedule(const GemmArgs &g, int sms) {
    return g.out == Dtype::FP32 && g.epilogue == Epilogue::Store ? weight_gradient_schedule(g, sms) : product_schedule(g, sms);
}

bool half_an_sm(const GemmArgs &g, const Schedule &sc, int sms) {
    const long long tiles = (long long)((g.m + BM - 1) / BM) * ((g.n + sc.bn - 1) / sc.bn) * g.batch;
    return g.beside_others && g.batch > 1 && g.out == Dtype::BF16 && (g.epilogue == Epilogue::Store || g.epilogue == Epilogue::Axpby) &&
           !sc.pair && sc.bn <= 128 && tiles * sc.splits <= sms;
}

// Scratch a schedule needs: FP32 partial tiles and one ticket per output tile (none without a K split).
struct ScratchNeed {
    size_t partial_bytes = 0, tickets = 0;
};
ScratchNeed scratch_need(const GemmArgs &g, const Schedule &sc) {
    if (sc.splits <= 1)
        return {};
    const int unit = sc.pair ? 2 : 1;
    const int m_tiles = (g.m + BM - 1) / BM, padded_m_tiles = (m_tiles + unit - 1) / unit * unit;
    const int n_tiles = (g.n + sc.bn - 1) / sc.bn;
    return {size_t(sc.splits) * g.batch * padded_m_tiles * BM * n_tiles * sc.bn * sizeof(float),
            size_t(padded_m_tiles) * n_tiles * g.batch};
}

// Stand-alone calls (tg_ex_gemm) share one workspace per device, grown on demand.
std::mutex shared_workspace_mutex;
std::unordered_map<int, GemmWorkspace> shared_workspaces;

void grow(GemmWorkspace &w, const ScratchNeed &need, cudaStream_t s) {
    if (!w.error_word) {
        CHECK_CUDA(cudaMalloc(&w.error_word, sizeof(StepCounters)));
        CHECK_CUDA(cudaMemset(w.error_word, 0, sizeof(StepCounters)));
    }
    if (w.partial_bytes < need.partial_bytes) {
        CHECK_CUDA(cudaStreamSynchronize(s));
        if (w.partials)
            CHECK_CUDA(cudaFree(w.partials));
        w.partials = nullptr, w.partial_bytes = 0;
        CHECK_CUDA(cudaMalloc(&w.partials, need.partial_bytes));
        w.partial_bytes = need.partial_bytes;
        ++w.generation;
    }
    if (w.ticket_count < need.tickets) {
        CHECK_CUDA(cudaStreamSynchronize(s));
        if (w.tickets)
            CHECK_CUDA(cudaFree(w.tickets));
        w.tickets = nullptr, w.ticket_count = 0;
        CHECK_CUDA(cudaMalloc(&w.tickets, need.tickets * sizeof(unsigned)));
        CHECK_CUDA(cudaMemset(w.tickets, 0, need.tickets * sizeof(unsigned)));
        w.ticket_count = need.tickets;
        ++w.generation;
    }
}

// The kernel counts work items in 32 bits.  Batches of more than this many go in several launches (one of 2^20 items takes milliseconds,
// so another costs nothing; K is whole there); a single matrix of more would not fit any memory.
constexpr long long MostItems = 1 << 20;

// Builds the kernel parameters and tensor maps for `sc` and launches.  `partials` / `tickets` may be
// null when the schedule does not split K.
void launch_schedule(const GemmArgs &g, const Schedule &sc, int sms, float *partials, unsigned *tickets,
                     StepCounters *counters, cudaStream_t s) {
    TcParams p{};
    p.m = g.m, p.n = g.n, p.k = g.k, p.batch = g.batch;
    p.a_mn = g.a_col == 1 ? 0 : 1;
    p.b_mn = g.b_col == 1 ? 0 : 1;
    p.epilogue = int(g.epilogue), p.out_fp32 = g.out == Dtype::FP32;
    p.bn = sc.bn, p.splits = sc.splits, p.k_blocks_per_split = sc.k_blocks_per_split;
    p.reduce_later = sc.splits >= 4; // K is only split for plain stores
    const int64_t lda = p.a_mn ? g.a_col : g.a_row, ldb = p.b_mn ? g.b_col : g.b_row;
    const int unit = sc.pair ? 2 : 1;
    const int m_tiles = (g.m + BM - 1) / BM, padded_m_tiles = (m_tiles + unit - 1) / unit * unit;
    const int n_tiles = (g.n + p.bn - 1) / p.bn;
    const long long matrix_tiles = (long long)(padded_m_tiles / unit) * n_tiles, tiles = matrix_tiles * g.batch; // scheduling units
    if (tiles > MostItems && g.batch > 1) {
        const int part = int(std::max(1ll, MostItems / matrix_tiles));
        auto at = [](const void *base, int64_t elements, Dtype t) { return base ? static_cast<const char *>(base) + elements * int64_t(dtype_size(t)) : nullptr; };
        for (int64_t z = 0; z < g.batch; z += part) {
            GemmArgs some = g;
            some.batch = int(std::min<int64_t>(part, g.batch - z));
            some.a = at(g.a, z * g.a_batch, g.in), some.b = at(g.b, z * g.b_batch, g.in), some.r = at(g.r, z * g.r_batch, g.out);
            some.c = const_cast<char *>(at(g.c, z * g.c_batch, g.out)), some.c2 = const_cast<char *>(at(g.c2, z * g.c_batch, g.out));
            launch_schedule(some, sc, sms, partials, tickets, counters, s);
        }
        return;
    }
    if (tiles > INT_MAX / 2)
        throw std::runtime_error("GEMM: too many tiles");
    const int bn_local = p.bn / unit;
    const int stage_bytes = StageABytes + bn_local * BK * 2;
    const int row_scratch = g.epilogue == Epilogue::CrossEntropy ? RowScratchBytes : 0;
    const bool half = half_an_sm(g, sc, sms);
    p.tmem_columns = half ? sc.bn : 2 * MaxBN;
    p.stages = ((half ? HalfShared : MaxShared) - 1024 - ControlBytes - row_scratch) / stage_bytes;
    if (p.stages > MaxStages)
        p.stages = MaxStages;
    const int shared = p.stages * stage_bytes + ControlBytes + row_scratch + 1024;
    p.c = g.c, p.c2 = g.c2, p.r = g.r;
    p.ldc = g.ldc, p.ldr = g.ldr, p.c_batch = g.c_batch, p.r_batch = g.r_batch;
    p.alpha = g.alpha, p.beta = g.beta;
    p.counters = counters;
    p.workspace = partials, p.tickets = tickets;
    {
        const int per32 = p.out_fp32 ? 8 : 16; // elements per 32 bytes
        auto aligned32 = [&](const void *ptr, int64_t ld, int64_t batch_stride) {
            return !ptr || (reinterpret_cast<uintptr_t>(ptr) % 32 == 0 && ld % per32 == 0 && batch_stride % per32 == 0);
        };
        p.wide = g.epilogue == Epilogue::CrossEntropy
                     ? aligned32(g.c, g.ldc, 0)
                     : aligned32(g.c, g.ldc, g.c_batch) && aligned32(g.c2, g.ldc, g.c_batch) && aligned32(g.r, g.ldr, g.r_batch);
    }
    CUtensorMap map_a = p.a_mn ? make_map_bf16(g.a, g.m, g.k, g.batch, lda, g.a_batch, 64, BK)
                               : make_map_bf16(g.a, g.k, g.m, g.batch, lda, g.a_batch, BK, BM);
    CUtensorMap map_b = p.b_mn ? make_map_bf16(g.b, g.n, g.k, g.batch, ldb, g.b_batch, 64, BK)
                               : make_map_bf16(g.b, g.k, g.n, g.batch, ldb, g.b_batch, BK, bn_local);
    const long long work = tiles * p.splits;
    const int slots = sms / unit;
    const int grid = int(work < slots ? work : slots) * unit;
    auto launch = [&](auto kernel) {
        // The opt-in shared-memory size is an attribute of each instantiation on each device.
        static std::mutex guard;
        static std::unordered_map<const void *, unsigned long long> configured; // kernel -> device bit mask
        int device = 0;
        CHECK_CUDA(cudaGetDevice(&device));
        {
            std::lock_guard<std::mutex> lock(guard);
            unsigned long long &mask = configured[reinterpret_cast<const void *>(kernel)];
            if (!(mask >> (device & 63) & 1ull)) {
                CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MaxShared));
                mask |= 1ull << (device & 63);
            }
        }
        cudaLaunchConfig_t config{};
        config.gridDim = dim3(grid), config.blockDim = dim3(threads_of(half ? 8 : 16));
        config.dynamicSmemBytes = shared, config.stream = s;
        cudaLaunchAttribute attributes[2]{};
        attributes[0].id = cudaLaunchAttributeClusterDimension;
        attributes[0].val.clusterDim.x = unit, attributes[0].val.clusterDim.y = 1, attributes[0].val.clusterDim.z = 1;
        // The kernel's set-up (barriers, tensor memory, descriptors) overlaps the tail of the kernel before it.
        attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attributes[1].val.programmaticStreamSerializationAllowed = 1;
        config.attrs = attributes, config.numAttrs = 2;
        CHECK_CUDA(cudaLaunchKernelEx(&config, kernel, map_a, map_b, p));
    };
    auto launch_kind = [&](auto pair_tag) {
        constexpr bool P = decltype(pair_tag)::value;
        if (p.out_fp32) {
            launch(gemm_tc_kernel<int(Epilogue::Store), true, P, 16>);
        } else {
            // A CTA's only tile: the product is hardly longer than the fetch of its weights, and most of that is hidden (tg_predict 12 layers d 768
            // 636 -> 624 us, 16 layers d 640, 74 tokens 572 -> 547, 2 layers d 896, 1381 tokens 187 -> 181).  With further tiles to come it is level or costs
            // more than it gives (evaluation of 6 layers d 512, 4096 tokens 366 -> 377), as it does in the training step, where the engine does not ask for
            // it (4 layers d 256, 2048 tokens: 343 -> 346 us a step).
            const bool early = g.b_settled && p.splits == 1 && work <= slots;
            switch (g.epilogue) {
            case Epilogue::Store:
                early ? launch(gemm_tc_kernel<int(Epilogue::Store), false, P, 16, true>) : launch(gemm_tc_kernel<int(Epilogue::Store), false, P, 16>);
                break;
            case Epilogue::Residual:
                early ? launch(gemm_tc_kernel<int(Epilogue::Residual), false, P, 16, true>) : launch(gemm_tc_kernel<int(Epilogue::Residual), false, P, 16>);
                break;
            case Epilogue::GeluDual: launch(gemm_tc_kernel<int(Epilogue::GeluDual), false, P, 16>); break;
            case Epilogue::Gelu:
                early ? launch(gemm_tc_kernel<int(Epilogue::Gelu), false, P, 16, true>) : launch(gemm_tc_kernel<int(Epilogue::Gelu), false, P, 16>);
                break;
            case Epilogue::GeluGrad: launch(gemm_tc_kernel<int(Epilogue::GeluGrad), false, P, 16>); break;
            case Epilogue::Axpby: launch(gemm_tc_kernel<int(Epilogue::Axpby), false, P, 16>); break;
            case Epilogue::CrossEntropy: launch(gemm_tc_kernel<int(Epilogue::CrossEntropy), false, P, 16>); break;
            }
        }
    };
    if (sc.pair)
        launch_kind(std::true_type{});
    else if (half && g.epilogue == Epilogue::Store)
        launch(gemm_tc_kernel<int(Epilogue::Store), false, false, 8>);
    else if (half)
        launch(gemm_tc_kernel<int(Epilogue::Axpby), false, false, 8>);
    else
        launch_kind(std::false_type{});
    CHECK_CUDA(cudaGetLastError());
    if (p.reduce_later) {
        const long long padded_m = (long long)padded_m_tiles * BM, padded_n = (long long)n_tiles * p.bn;
        const unsigned blocks = unsigned(padded_m / 32 * (padded_n / 32) * g.batch);
        if (p.out_fp32)
            splitk_reduce_kernel<true><<<blocks, 256, 0, s>>>(p, padded_m, padded_n);
        else
            splitk_reduce_kernel<false><<<blocks, 256, 0, s>>>(p, padded_m, padded_n);
        CHECK_CUDA(cudaGetLastError());
    }
}
} // namespace

int gemm_tc_shared_bytes() { return MaxShared; }

bool gemm_tc_supported(const GemmArgs &g) {
    if (g.in != Dtype::BF16)
        return false;
    if (g.m < 1 || g.n < 64 || g.k < 64 || g.n % 8)
        return false;
    const bool a_k = g.a_col == 1, a_mn = g.a_row == 1, b_k = g.b_col == 1, b_mn = g.b_row == 1;
    if (!(a_k || a_mn) || !(b_k || b_mn))
        return false;
    const int64_t lda = a_k ? g.a_row : g.a_col, ldb = b_k ? g.b_row : g.b_col;
    if (lda % 8 || ldb % 8 || g.ldc % 8 || (g.r && g.ldr % 8))
        return false;
    const bool loss = g.epilogue == Epilogue::CrossEntropy; // R holds one byte per row there
    if (loss && (g.n != 256 || g.batch != 1 || g.out != Dtype::BF16 || !g.r || !g.c2 || g.a_col != 1 || g.b_col != 1))
        return false;
    if (reinterpret_cast<uintptr_t>(g.a) % 16 || reinterpret_cast<uintptr_t>(g.b) % 16 ||
        reinterpret_cast<uintptr_t>(g.c) % 16 || (!loss && reinterpret_cast<uintptr_t>(g.r) % 16) ||
        reinterpret_cast<uintptr_t>(g.c2) % 16)
        return false;
    if (g.a_batch % 8 || g.b_batch % 8 || g.c_batch % 8 || g.r_batch % 8)
        return false;
    if (g.out == Dtype::FP32 && g.epilogue != Epilogue::Store)
        return false;
    return true;
}

namespace {
void launch_with(const GemmArgs &g, const Schedule &sc, int sms, StepCounters *counters, cudaStream_t s,
                 GemmWorkspace *workspace);
}

void release_gemm_workspace(GemmWorkspace &w) {
    if (w.partials)
        cudaFree(w.partials);
    if (w.tickets)
        cudaFree(w.tickets);
    if (w.error_word)
        cudaFree(w.error_word);
    w = GemmWorkspace{};
}

// `workspace`: the caller's own split-K scratch (an Engine's: grown here, outside stream capture,
// when a schedule needs more); nullptr: the per-device workspace shared by the stand-alone calls,
// whose device-side give-ups are reported by gemm_tc_take_device_error().
int launch_gemm_tc(const GemmArgs &g, int sms, StepCounters *counters, cudaStream_t s, GemmWorkspace *workspace) {
    const Schedule sc = choose_schedule(g, sms);
    launch_with(g, sc, sms, counters, s, workspace);
    return sc.splits >= 4 ? 2 : 1; // the product kernel, and the kernel that adds many splits' partial tiles
}

namespace {
void launch_with(const GemmArgs &g, const Schedule &sc, int sms, StepCounters *counters, cudaStream_t s,
                 GemmWorkspace *workspace) {
    const ScratchNeed need = scratch_need(g, sc);
    if (workspace) {
        if (need.partial_bytes > workspace->partial_bytes || need.tickets > workspace->ticket_count || !workspace->error_word)
            grow(*workspace, need, s);
        launch_schedule(g, sc, sms, workspace->partials, workspace->tickets, counters, s);
        return;
    }
    int device = 0;
    CHECK_CUDA(cudaGetDevice(&device));
    std::lock_guard<std::mutex> lock(shared_workspace_mutex);
    GemmWorkspace &w = shared_workspaces[device];
    grow(w, need, s);
    launch_schedule(g, sc, sms, w.partials, w.tickets, counters ? counters : w.error_word, s);
}
} // namespace

// ------------------------------------------------------------------------------------------
// Weight gradient without any allocation.  Some hosts may not call cudaMalloc at the moment they
// need a gradient: a serving or training process that has handed the whole device to its own
// memory pool, a caller inside a region where the allocator's implicit device synchronisation is
// not acceptable, or one whose memory budget was fixed when the process started.  For them the
// split-K scratch (FP32 partial tiles, the per-tile tickets and a device error word) lives in the
// array below, which every GPU that loads this library holds until the process exits.
//
// In host code `static_scratch` is only a stand-in for the symbol: its device address comes from
// cudaGetSymbolAddress, fetched once per device with that device current, on the first call for
// that device (so the first call should happen before any stream capture).  All calls share the
// array and it keeps the previous call's contents: the tickets are cleared on the stream before
// every launch, the partial tiles are fully overwritten before they are read.  Two calls that
// overlap on the GPU (different streams, or different threads) race on it.
//
// The schedule (tile width, K splits, CTA pair) and the kernel are exactly those tg_ex_gemm uses
// for the same shape, so the results are bit-identical to it.
// ------------------------------------------------------------------------------------------
namespace {
constexpr size_t StaticPartialBytes = size_t(16) << 20; // 16 MiB of FP32 partial tiles
constexpr int StaticTickets = 1024;                      // output tiles
constexpr size_t StaticErrorOffset = StaticPartialBytes + StaticTickets * sizeof(unsigned);
static __device__ __align__(256) unsigned char static_scratch[StaticErrorOffset + 256];
void *static_scratch_address[64] = {}; // per device, filled on first use
} // namespace

GemmSchedule gemm_tc_schedule(const GemmArgs &g, int sms) {
    const Schedule sc = choose_schedule(g, sms);
    return {sc.bn, sc.splits, sc.pair, half_an_sm(g, sc, sms)};
}
size_t gemm_tc_static_scratch_bytes() { return StaticPartialBytes; }

void launch_weight_gradient_static(const void *dy, const void *x, float *dw, int out, int in, int tokens,
                                   int sms, cudaStream_t s) {
    // dW[out, in] = dy[tokens, out]^T x[tokens, in]: both operands MN-major, K = tokens.
    GemmArgs g;
    g.in = Dtype::BF16, g.out = Dtype::FP32;
    g.a = dy, g.a_row = 1, g.a_col = out, g.b = x, g.b_row = 1, g.b_col = in;
    g.c = dw, g.ldc = in, g.m = out, g.n = in, g.k = tokens;
    if (!gemm_tc_supported(g))
        throw std::runtime_error("weight gradient: sizes must be multiples of 8 (out, in), at least 64, and the "
                                 "pointers 16-byte aligned");
    int device = 0;
    CHECK_CUDA(cudaGetDevice(&device));
    if (device < 0 || device >= 64)
        throw std::runtime_error("weight gradient: device index out of range");
    if (!static_scratch_address[device]) { // set-up, once per device, with that device current
        void *address = nullptr;
        CHECK_CUDA(cudaGetSymbolAddress(&address, static_scratch));
        CHECK_CUDA(cudaMemsetAsync(static_cast<unsigned char *>(address) + StaticErrorOffset, 0, 256, s));
        static_scratch_address[device] = address;
    }
    const Schedule sc = choose_schedule(g, sms);
    const ScratchNeed need = scratch_need(g, sc);
    if (need.partial_bytes > StaticPartialBytes || need.tickets > size_t(StaticTickets))
        throw std::runtime_error("weight gradient: this shape needs " + std::to_string(need.partial_bytes) +
                                 " bytes of scratch in " + std::to_string(need.tickets) +
                                 " tiles; the built-in array holds " + std::to_string(StaticPartialBytes) +
                                 " bytes and " + std::to_string(StaticTickets) + " tiles (use tg_ex_gemm, which allocates)");
    unsigned char *scratch = static_cast<unsigned char *>(static_scratch_address[device]);
    unsigned *tickets = reinterpret_cast<unsigned *>(scratch + StaticPartialBytes);
    CHECK_CUDA(cudaMemsetAsync(tickets, 0, StaticTickets * sizeof(unsigned), s)); // must start at zero
    launch_schedule(g, sc, sms, reinterpret_cast<float *>(scratch), tickets,
                    reinterpret_cast<StepCounters *>(scratch + StaticErrorOffset), s);
}

// First device-side give-up code recorded by the stand-alone calls (tg_ex_gemm, tg_ex_head_cross_entropy,
// tg_ex_weight_gradient_static, attention) on the current device since the last query; 0 when none.
// Synchronises `s`; allocates nothing.
int gemm_tc_take_device_error(cudaStream_t s) {
    int device = 0;
    CHECK_CUDA(cudaGetDevice(&device));
    CHECK_CUDA(cudaStreamSynchronize(s));
    StepCounters *words[3] = {nullptr, nullptr, attention_error_word(false)};
    {
        std::lock_guard<std::mutex> lock(shared_workspace_mutex);
        auto found = shared_workspaces.find(device);
        if (found != shared_workspaces.end())
            words[0] = found->second.error_word;
    }
    if (device >= 0 && device < 64 && static_scratch_address[device])
        words[1] = reinterpret_cast<StepCounters *>(static_cast<unsigned char *>(static_scratch_address[device]) +
                                                    StaticErrorOffset);
    int code = 0;
    for (StepCounters *word : words) {
        if (!word)
            continue;
        StepCounters host{};
        CHECK_CUDA(cudaMemcpy(&host, word, sizeof(host), cudaMemcpyDeviceToHost));
        if (host.error) {
            if (!code)
                code = host.error;
            CHECK_CUDA(cudaMemset(word, 0, sizeof(StepCounters)));
        }
    }
    return code;
}
