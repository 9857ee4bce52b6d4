// How the epilogues of tensor-core products touch global memory: a lane drains its own row of tensor memory, pairs of lanes
// exchange halves of their rows before they store (and after they load).
#pragma once
#include <cstdint>

// Two neighbouring lanes hold a row each, eight words (32 bytes) at `low` and eight at `high`: afterwards `low` is the even lane's row
// and `high` the odd lane's, the first 32 bytes of them in the even lane and the second in the odd one.  A warp's 256-bit access then
// touches 16 pieces of 64 bytes.  With lane = row, 32 pieces of 32 bytes, stores run at 18 B/clk and SM and loads at 32 where the
// paths from and to L2 carry 32 and 64; measured 3710 and 2050 clocks for a 128 x 256 tile's stores, 2060 and 1060 for loads.  As much
// as the pairs gives whole lines: four lanes exchanged through twice the shuffles stored no faster.
__device__ __forceinline__ void exchange_rows(uint32_t *low, uint32_t *high, bool odd) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? low[j] : high[j], 1);
        low[j] = odd ? got : low[j];
        high[j] = odd ? high[j] : got;
    }
}

// 32 bytes to or from global memory: one 256-bit access when `wide` (32-byte aligned), else two
// 128-bit accesses; `second` says whether the upper half is inside the tensor.
__device__ __forceinline__ void load_global32(const void *p, uint32_t (&r)[8], bool wide, bool second) {
    if (wide) {
        asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "l"(p));
    } else {
        uint4 a = *reinterpret_cast<const uint4 *>(p), b = make_uint4(0, 0, 0, 0);
        if (second)
            b = *(reinterpret_cast<const uint4 *>(p) + 1);
        r[0] = a.x, r[1] = a.y, r[2] = a.z, r[3] = a.w, r[4] = b.x, r[5] = b.y, r[6] = b.z, r[7] = b.w;
    }
}
__device__ __forceinline__ void store_global32(void *p, const uint32_t *r, bool wide, bool second) {
    if (wide) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(r[0]), "r"(r[1]),
                     "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                     : "memory");
    } else {
        *reinterpret_cast<uint4 *>(p) = make_uint4(r[0], r[1], r[2], r[3]);
        if (second)
            *(reinterpret_cast<uint4 *>(p) + 1) = make_uint4(r[4], r[5], r[6], r[7]);
    }
}
