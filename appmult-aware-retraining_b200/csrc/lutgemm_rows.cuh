// Shared-memory table and slab build of the kernels in which a thread owns whole output rows (lutgemm_slab_rows.cu,
// lutgemm_forward_rows.cu): tables turned to rows of one column (term) code, and slabs of 128-byte rows - 64 entries of 16 bits - one
// per row code.
#pragma once

#include "lutgemm_common.cuh"

namespace lutgemm {

template <int BITS>
struct RowsTable {
    static constexpr int Q = 1 << BITS;
    static constexpr int ROW = BITS == 4 ? 36 : 2 * Q;  // bytes per table row (4 bits: padded, rows on different banks)
    static constexpr int BYTES = (Q * ROW + 127) & ~127;
    static constexpr int U_ROW = 128, U_BYTES = Q * U_ROW;  // slab
    // turning passes the wire-format table through a buffer, TURN_ROWS of its rows at a time
    static constexpr int TURN_ROWS = BITS == 8 ? 128 : Q, TURN_BYTES = TURN_ROWS * lut_col_num(BITS) * 2;
};

// table[y][x] = lut[x * COL + y] ^ flip for 512 threads.  The rows of the wire format have an odd number of words, so reading
// columns of the copy in `buffer` is free of bank conflicts, as are the stores.  The caller synchronises before and after.
template <int BITS>
__device__ __forceinline__ void stage_table_turned(uint8_t *table, uint8_t *buffer, const uint16_t *__restrict__ lut, uint32_t flip, int tid) {
    using T = RowsTable<BITS>;
    constexpr int COL = lut_col_num(BITS), THREADS = 512;
    uint16_t *raw = reinterpret_cast<uint16_t *>(buffer);
    const bool vec = (reinterpret_cast<uintptr_t>(lut) & 15) == 0;
    static_assert(T::TURN_ROWS == T::Q || T::TURN_ROWS * COL % 8 == 0, "the second half is as aligned as the first");
#pragma unroll 1
    for (int x0 = 0; x0 < T::Q; x0 += T::TURN_ROWS) {
        const uint16_t *src = lut + x0 * COL;
        if (x0) __syncthreads();
        if (vec) {
            constexpr int VECS = T::TURN_BYTES / 16;
            for (int idx = tid; idx < VECS; idx += THREADS) cp_async16(raw + 8 * idx, src + 8 * idx);
            for (int idx = 8 * VECS + tid; idx < T::TURN_ROWS * COL; idx += THREADS) raw[idx] = src[idx];
            cp_async_commit();
            cp_async_wait<0>();
        } else {
#pragma unroll 8
            for (int idx = tid; idx < T::TURN_ROWS * COL; idx += THREADS) raw[idx] = src[idx];
        }
        __syncthreads();
#pragma unroll 4
        for (int idx = tid; idx < T::TURN_ROWS / 2 * T::Q; idx += THREADS) {
            const int xp = idx % (T::TURN_ROWS / 2), y = idx / (T::TURN_ROWS / 2);
            const uint32_t e0 = raw[2 * xp * COL + y], e1 = raw[(2 * xp + 1) * COL + y];
            *reinterpret_cast<uint32_t *>(table + y * T::ROW + (x0 + 2 * xp) * 2) = (e0 | e1 << 16) ^ flip;
        }
    }
}

// table[x][y] = lut[x * COL + y] ^ flip, rows as they are
template <int BITS>
__device__ __forceinline__ void stage_table_plain(uint8_t *table, const uint16_t *__restrict__ lut, uint32_t flip, int tid) {
    using T = RowsTable<BITS>;
    constexpr int COL = lut_col_num(BITS), Q = T::Q, THREADS = 512;
    if ((reinterpret_cast<uintptr_t>(lut) & 3u) == 0) {  // (COL is even: pairs of entries are 4-byte aligned)
        const uint32_t *src = reinterpret_cast<const uint32_t *>(lut);
#pragma unroll 8
        for (int idx = tid; idx < Q * Q / 2; idx += THREADS)
            *reinterpret_cast<uint32_t *>(table + idx / (Q / 2) * T::ROW + idx % (Q / 2) * 4) = src[idx / (Q / 2) * (COL / 2) + idx % (Q / 2)] ^ flip;
    } else {
        for (int idx = tid; idx < Q * Q; idx += THREADS)
            *reinterpret_cast<uint16_t *>(table + (idx >> BITS) * T::ROW + (idx & (Q - 1)) * 2) =
                lut[(idx >> BITS) * COL + (idx & (Q - 1))] ^ (uint16_t)flip;
    }
}

// A thread's share of a slab build by 512 threads: four columns (quad bq) x eight codes (16 bytes of a table row; four codes at
// 6 bits, one at 4).  One step builds a slab at 8 bits, two at fewer.  The lanes are staggered over the table rows' chunks, so
// that reads are free of bank conflicts whatever the column codes are, and a half-warp stores sixteen different quads.
template <int BITS>
struct SlabBuild {
    using T = RowsTable<BITS>;
    uint32_t table, slab;  // shared addresses: the thread's first code in table row 0 and in slab row 0 of the unit at u_addr
    int codes;             // offset of its four column codes
    __device__ __forceinline__ SlabBuild(uint32_t tt_addr, uint32_t u_addr, int tid) {
        const int bq = tid & 15, hx = tid >> 4, bs = BITS < 8 ? hx >> 4 : 0;
        const int bx = BITS == 8 ? (hx ^ (bq & 7)) * 8 : BITS == 7 ? ((hx & 15) ^ (bq & 7)) * 8 : BITS == 6 ? ((hx & 15) ^ bq) * 4 : hx & 15;
        table = tt_addr + bx * 2;
        slab = u_addr + bs * T::U_BYTES + bx * T::U_ROW + bq * 8;
        codes = bs * 64 + bq * 4;
    }
    // slabs at byte offset `off` of the buffers, from 64 column codes each
    __device__ __forceinline__ void step(uint32_t off, const uint8_t *cc) const {
        const uint32_t cw = *reinterpret_cast<const uint32_t *>(cc + codes);
        uint32_t ad[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) ad[c] = table + byte_of(cw, c) * T::ROW;
        const uint32_t ub = slab + off;
        auto put = [&](int row, uint32_t lo, uint32_t hi) {
            asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(ub + row * T::U_ROW), "r"(lo), "r"(hi) : "memory");
        };
        if constexpr (BITS >= 6) {
            constexpr int W = BITS == 6 ? 2 : 4;
            uint32_t r[4][W];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if constexpr (W == 4)
                    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(r[c][0]), "=r"(r[c][1]), "=r"(r[c][W - 2]), "=r"(r[c][W - 1]) : "r"(ad[c]));
                else
                    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(r[c][0]), "=r"(r[c][1]) : "r"(ad[c]));
            }
#pragma unroll
            for (int e = 0; e < 2 * W; ++e) {
                const uint32_t sel = e & 1 ? 0x7632u : 0x5410u;
                put(e, __byte_perm(r[0][e / 2], r[1][e / 2], sel), __byte_perm(r[2][e / 2], r[3][e / 2], sel));
            }
        } else {
            uint32_t r[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) r[c] = lds_u16(ad[c]);
            put(0, r[0] | r[1] << 16, r[2] | r[3] << 16);
        }
    }
};

}  // namespace lutgemm
