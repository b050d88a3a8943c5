// Gradient LUT-GEMM kernel for sm_100a, one thread per output row: tiles of 512 rows x 64 terms.
//
//   grad_a:  ga[m,k] = 1/16 * sum_n gc[m,n] * T(a[m,k], w[k,n])     rows r = m, terms = n
//   grad_x:  gx[b,c,h,w] = 1/16 * sum_{taps (i,j)} sum_n gy[m(b,h,w,i,j), n] * T(x[b,c,h,w], wmat[(c,i,j), n])
//            rows r = input pixels, terms = (tap, n), the k loop runs over the input channels c
//   grad_w:  gw[k,n] = 1/16 * sum_m T(a[m,k], w[k,n]) * gc[m,n]     rows r = n, terms = m
//
// Per k a slab U_k[x][t] = T(x, code[k,t]) is gathered once for all 2^b row codes x and the 64 terms of the tile.  A
// thread owns one output row and keeps the row's 64 grad_out values in registers for the whole k loop; for every k it
// reads the slab row of its own code and takes the dot product, so the sum over the terms stays inside the thread: no
// partial sums of one k are exchanged between threads or warps.
//
// Bank conflicts: a slab row is 128 bytes, eight 16-byte chunks that lie in the same bank quads for every row code.  Lane l
// reads its chunks in the order j ^ (l & 7), so the eight lanes of a quarter-warp are on eight different quads whatever
// their codes are; the grad_out registers are loaded in the same order, so nothing is indexed at run time.
// The build reads the table (rows of one column code contiguous in x) in 16-byte pieces, lanes staggered the same way, and
// stores four terms of one code at a time, each half-warp on sixteen different bank pairs: reads and stores are
// conflict-free too.
//
// From 16-bit entries to products, two at a time: the table is staged in offset-binary, each half of a slab word goes behind
// the exponent of 2^23 (a byte permutation), one packed subtraction of 2^23 + 2^15 leaves the two signed entries exactly, and one
// packed multiply-add (fma.rn.f32x2) consumes them.  Entries that are zero add nothing, whatever else the table holds.  With
// an offset left in the entries and taken off the sum (their bits as subnormal floats: 9.06 ms instead of 9.74 at 4096^3 and 7 bits)
// sums of small entries keep the rounding errors of the offset: sparse codes, of which 99 % are zero, were off by up to 3.5e-6.
// Errors against 64-bit sums, 2-norm, 4 to 8 bits, 320 to 60000 terms: 0.9e-7 to 1.1e-7 for uniform codes, less where half of them and
// more are zero (with terms across lanes, lutgemm_slab_grad.cu, 0.8e-7 to 1.0e-7).
//
// What bounds it: instruction issue, as a packed fp32 instruction takes two slots.  7 bits, 4096 x 512 x 4096, per k and tile (32768
// look-ups): 3390 warp instructions, 1060 of them packed, 1250 clocks: 90 % of the issue slots; 810 shared-memory wavefronts,
// 62 % of that pipe.  8 bits: 4100 instructions, 1100 wavefronts, 1535 clocks.  grad_w / grad_a of 4096^3 against the kernel with terms
// across lanes: 8 bits 14.15 / 14.95 -> 11.76 / 11.77 ms, 7 bits 9.99 / 10.09 -> 9.76 / 9.77, 6 bits 9.62 / 9.63 -> 9.64 / 9.67; grad_x: 3x3,
// 64 channels at 32 x 32, batch 256, 7 bits 1.80 -> 1.47 ms; 1x1, 256 -> 64 channels at 56 x 56, batch 64, 8 bits, 1.44 (broadcast) -> 0.56.
//
// Of the 128 registers that 512 threads leave a thread, grad_out takes 64: grad_x spills 16 bytes at 4, 6 and 8 bits, the others none.
//
// A CTA takes the term blocks of a group one after the other and adds each to the group's sums.  More than kRowsChain
// blocks are added in two levels (blocks of a run of kRowsRun into a buffer of the CTA, runs into the group's sums), so that
// no chain of additions grows with the problem by more than one per 512 terms.  The same thread stores, adds and reads
// a sum, so nothing needs ordering between threads and results are deterministic.
// Every wait on a barrier is bounded (lutgemm_waits.cuh).
// Replaces ApproxGemmBackwardKernelForGA / ForGB, self_ops/src/approx_gemm_backward.cu:13-258, 261-492, and for
// grad_x the unfold backward of self_ops/ops_py/approx_ops.py:556-571.
#include "lutgemm_common.cuh"
#include "lutgemm_f32x2.cuh"
#include "lutgemm_kernels.h"
#include "lutgemm_rows.cuh"
#include "lutgemm_waits.cuh"

namespace lutgemm {
namespace sr {

enum { kGw = 1, kGa = 2, kGx = 3 };

template <int BITS>
struct Cfg {
    static constexpr int Q = 1 << BITS;
    static constexpr int WARPS = 16, THREADS = 512, RT = kRowsTile, CT = kRowsTerms;
    static constexpr int KC = 16;                        // k per operand stage
    // k per unit - what the warps hand over to each other - as many as fit three times: grad_w / grad_a of 4096^3 at 7 bits 9.75 /
    // 9.75 ms with four, 9.96 / 10.24 with two; at 8 bits there is room for one
    static constexpr int KU = BITS == 8 ? 1 : 4, NB = 3;
    using T = RowsTable<BITS>;
    static constexpr int TT_ROW = T::ROW, TT_BYTES = T::BYTES, U_ROW = T::U_ROW, U_BYTES = T::U_BYTES, UB = KU * U_BYTES;
    static constexpr int CC_STAGE = KC * CT;
    static constexpr int OFF_U = TT_BYTES;
    // a block's grad_out values pass through the slab buffers, G_ROWS rows at a time, with grad_x's pixels behind them
    static constexpr int G_ROWS = NB * UB >= RT * CT * 4 + RT * 8 ? RT : RT / 2;
    static constexpr int G_BYTES = G_ROWS * CT * 4;
    static constexpr int OFF_CC = OFF_U + (NB * UB > G_BYTES + RT * 8 ? NB * UB : G_BYTES + RT * 8);
    static constexpr int OFF_BAR = OFF_CC + 2 * CC_STAGE;
    static constexpr int OFF_TAP = OFF_BAR + NB * 8 + 8;  // behind an mbarrier per buffer and the abort word
    static constexpr int SMEM = OFF_TAP + kMaxTaps * 2;  // grad_x: output offset {rows, columns} of each tap
    static_assert(U_ROW == 2 * CT && OFF_U % 128 == 0, "chunks of a slab row lie on fixed bank quads");
    static_assert(SMEM <= 232448, "shared memory budget");
    static_assert(T::TURN_BYTES <= NB * UB, "the table passes through the slab buffers");
};

struct Args {
    const uint8_t *rows;      // row codes: code of row r for k at rows[row_offset(r) + k * row_stride]
    const uint8_t *cols;      // term codes: grad_a w[k][n], grad_w at[k][m], grad_x wmat
    const int16_t *lut;
    const float *gc;
    float *out;
    float *tmp;               // per CTA: sums of a run of term blocks, [k of the item][row]
    long row_stride;
    long col_pitch;           // grad_a: N; grad_w: at_pitch
    int M, K, N;              // kGx: M = pixels of the class (all images), K = channels, N = Cout
    int RDIM, TDIM;           // rows and terms
    int tiles;
    RowsPlan plan;
    int direct;               // one group, and its sums go to their final place
    int vec_c, vec_g;
    int *error_word;
    PixelClass px;            // kGx only
};

// stores v or adds it to what is there, as a predicated instruction
template <bool ADD>
__device__ __forceinline__ void put(float *dst, float v, bool pred) {
    if (ADD)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p red.global.add.f32 [%0], %1;\n\t}" ::"l"(dst), "f"(v), "r"((uint32_t)pred) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.global.f32 [%0], %1;\n\t}" ::"l"(dst), "f"(v), "r"((uint32_t)pred) : "memory");
}

template <int BITS, int MODE>
__global__ void __launch_bounds__(512, 1) slab_grad_rows_kernel(const __grid_constant__ Args p) {
    using C = Cfg<BITS>;
    constexpr int Q = C::Q, RT = C::RT, CT = C::CT, KC = C::KC, KU = C::KU, NB = C::NB, UB = C::UB, THREADS = C::THREADS;
    constexpr uint32_t MASK4 = (Q - 1) * 0x01010101u;
    const int K = p.K, N = p.N;

    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t *cc_s = smem + C::OFF_CC;
    char2 *tap_s = reinterpret_cast<char2 *>(smem + C::OFF_TAP);
    const uint32_t tt_addr = smem_u32(smem), u_addr = smem_u32(smem + C::OFF_U);
    const uint32_t bar_full = smem_u32(smem + C::OFF_BAR);
    volatile int *abort_word = reinterpret_cast<volatile int *>(smem + C::OFF_BAR + 8 * NB);
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5, l7 = lane & 7;

    // ---- stage the gradient table in offset-binary: tt[y][x], x = row code, y = term code, T = lut[a * COL + w] -----------
    // (grad_w: rows are weight codes; grad_a / grad_x: rows are activation codes, so the table is turned)
    const uint16_t *lut = reinterpret_cast<const uint16_t *>(p.lut);
    if (MODE == kGw) stage_table_plain<BITS>(smem, lut, 0x80008000u, tid);
    else stage_table_turned<BITS>(smem, smem + C::OFF_U, lut, 0x80008000u, tid);
    if (tid == 0) *abort_word = 0;
    if (tid < 2 * C::CC_STAGE / 16) reinterpret_cast<uint4 *>(cc_s)[tid] = make_uint4(0, 0, 0, 0);  // (codes past the last k)
    if (MODE == kGx) {
        // pixel (hh, ww) of the class sits at h = ph + s hh; tap q connects it to output row (h - dh) / s = hh + eh
        for (int q = tid; q < p.px.ntaps; q += THREADS)
            tap_s[q] = make_char2((p.px.ph - p.px.dh[q]) / p.px.s, (p.px.pw - p.px.dw[q]) / p.px.s);
    }

    // ---- term codes: 16 k x 64 terms per stage, one 16-byte vector for each of the first 64 threads ---------------------
    auto load16 = [&](const uint8_t *src, int valid) -> uint4 {  // up to 16 bytes, the rest 0
        uint32_t t[4] = {0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < 16; ++q)
            if (q < valid) t[q >> 2] |= (uint32_t)src[q] << (8 * (q & 3));
        return make_uint4(t[0], t[1], t[2], t[3]);
    };
    auto col_codes16 = [&](int k, int t) -> uint4 {  // terms t .. t + 15 of k
        if (k >= K || t >= p.TDIM) return make_uint4(0, 0, 0, 0);
        if (MODE != kGx) {
            const uint8_t *src = p.cols + (size_t)k * p.col_pitch + t;
            return p.vec_c ? *reinterpret_cast<const uint4 *>(src) : load16(src, min(16, p.TDIM - t));
        }
        int q = t / N, n = t - q * N;
        if (p.vec_c)  // N % 16 == 0: the 16 terms lie inside one tap
            return *reinterpret_cast<const uint4 *>(p.cols + ((size_t)k * p.px.T + p.px.t[q]) * N + n);
        uint32_t v[4] = {0, 0, 0, 0};
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (t + i < p.TDIM) v[i >> 2] |= (uint32_t)p.cols[((size_t)k * p.px.T + p.px.t[q]) * N + n] << (8 * (i & 3));
            if (++n == N) { n = 0; ++q; }
        }
        return make_uint4(v[0], v[1], v[2], v[3]);
    };
    uint4 pcc = make_uint4(0, 0, 0, 0);
    auto fetch_cols = [&](int t0, int kbase) {
        if (tid < KC * CT / 16) pcc = col_codes16(kbase + tid / (CT / 16), t0 + (tid % (CT / 16)) * 16);
    };
    auto store_cols = [&](int stage) {
        if (tid < KC * CT / 16)
            *reinterpret_cast<uint4 *>(cc_s + stage * C::CC_STAGE + tid * 16) =
                make_uint4(pcc.x & MASK4, pcc.y & MASK4, pcc.z & MASK4, pcc.w & MASK4);
    };

    const SlabBuild<BITS> builder(tt_addr, u_addr, tid);
    auto build = [&](uint32_t off, const uint8_t *codes) {  // codes of the unit's first k
#pragma unroll
        for (int i = 0; i < (KU + 1) / 2; ++i) builder.step(off + i * 2 * C::U_BYTES, codes + i * 2 * CT);
    };

    const f32x2 bias = pack2(-8421376.0f, -8421376.0f);  // -(2^23 + 2^15)
    const f32x2 minus_zero = pack2(-0.0f, -0.0f);
    const uint32_t ul = u_addr + (l7 << 4);
    const float factor = p.direct ? kGradFactor : 1.0f;
    const RowsPlan &pl = p.plan;
    const int kunits = (K + kRowsUnit - 1) / kRowsUnit;
    const long total = (long)p.tiles * pl.groups * kunits;
    int cur = (int)(total * blockIdx.x / gridDim.x);  // (the launch checks that units can be counted in 32 bits)
    const int cur_end = (int)(total * (blockIdx.x + 1) / gridDim.x);
    bool first_block = true;
    while (cur < cur_end) {
        const int cell = cur / kunits, k0 = cur - cell * kunits;
        const int group = cell % pl.groups, tile = cell / pl.groups;
        const int nk = min(min(cur_end - cur, kunits - k0), pl.piece_k / kRowsUnit);
        const int kbeg = k0 * kRowsUnit, kend = min(K, (k0 + nk) * kRowsUnit);
        cur += nk;
        const int nblocks = min(pl.group_blocks, (p.TDIM + CT - 1) / CT - group * pl.group_blocks);
        const int row = tile * RT + tid, rowc = min(row, p.RDIM - 1);
        const bool in = row < p.RDIM;
        const size_t ostride = MODE == kGx && p.direct ? (size_t)p.px.H * p.px.W : (size_t)p.RDIM;
        const uint32_t roff = MODE == kGx ? (uint32_t)pixel_class_offset(p.px, rowc) : (uint32_t)rowc;
        const uint32_t ooff = MODE == kGx && p.direct ? roff : (uint32_t)rowc;
        const uint8_t *rows0 = p.rows + (size_t)kbeg * p.row_stride;
        float *out0 = p.out + (p.direct ? (size_t)0 : (size_t)group * K * p.RDIM) + (size_t)kbeg * ostride;
        float *tmp0 = p.tmp + (size_t)blockIdx.x * pl.piece_k * RT;  // (used with two_level only)
        const bool two_level = nblocks > kRowsChain;

#pragma unroll 1
        for (int block = 0; block < nblocks; ++block) {
            const int t0 = (group * pl.group_blocks + block) * CT;
            fetch_cols(t0, kbeg);
            // the row's codes of four k at a time, fetched one group ahead
            const uint8_t *rp = rows0;
            uint32_t raw[4];
            auto fetch_rows = [&](int k) {
#pragma unroll
                for (int i = 0; i < 4; ++i) raw[i] = k + i < kend ? (rp + i * p.row_stride)[roff] : 0u;
                rp += 4 * p.row_stride;
            };
            fetch_rows(kbeg);

            // The row's grad_out values of this block: g[4 j + w] = terms 2 w and 2 w + 1 of chunk j ^ l7.  They come through
            // shared memory: read by the threads themselves, every load touches as many cache lines as a warp has rows
            // (a block of 3x3 taps of 64 channels cost 17500 clocks beyond its k steps, now 9000)
            f32x2 g[32];
            float *g_s = reinterpret_cast<float *>(smem + C::OFF_U);
            int2 *pix_s = reinterpret_cast<int2 *>(smem + C::OFF_U + C::G_BYTES);  // grad_x: output position of tap offset 0, pixel
            constexpr int GR = C::G_ROWS;
            __syncthreads();  // the block before (or the table staging) is done with every buffer
            if (MODE == kGx) {
                const int perimg = p.px.Hc * p.px.Wc, b = rowc / perimg, rr = rowc - b * perimg, hh = rr / p.px.Wc, ww = rr - hh * p.px.Wc;
                pix_s[tid] = in ? make_int2((b * p.px.Ho + hh) * p.px.Wo + ww, hh << 16 | ww) : make_int2(0, -1);
                __syncthreads();
            }
#pragma unroll 1
            for (int r0 = 0; r0 < RT; r0 += GR) {
                if (r0) __syncthreads();
                if (MODE == kGw) {
                    // [term][row]
                    if (p.vec_g) {
#pragma unroll
                        for (int i = 0; i < CT * GR / 4 / THREADS; ++i) {
                            const int t = tid / (GR / 4) + THREADS / (GR / 4) * i, c = tid % (GR / 4) * 4, n = tile * RT + r0 + c;
                            const bool valid = t0 + t < p.M && n < N;  // N % 4 == 0
                            cp_async16_zfill(g_s + t * GR + c, valid ? p.gc + (size_t)(t0 + t) * N + n : p.gc, valid);
                        }
                    } else {
#pragma unroll 8
                        for (int i = 0; i < CT * GR / THREADS; ++i) {
                            const int t = tid / GR + THREADS / GR * i, c = tid % GR, n = tile * RT + r0 + c;
                            g_s[t * GR + c] = t0 + t < p.M && n < N ? p.gc[(size_t)(t0 + t) * N + n] : 0.f;
                        }
                    }
                } else {
                    // [row][term], the 16-byte pieces of rows 4 - 7 of eight swapped in pairs (no bank conflicts when read)
                    const int per = p.vec_g ? 4 : 1, pieces = CT / per;  // (N % 4 == 0: the four terms of a piece share their tap)
                    const int c = tid % pieces * per, t = t0 + c;
                    const int tap = MODE == kGx ? t / N : 0, n = t - tap * N;
                    int dh = 0, dw = 0;
                    if (MODE == kGx && t < p.TDIM) {
                        const char2 o = tap_s[tap];
                        dh = o.x;
                        dw = o.y;
                    }
                    auto src_of = [&](int r) -> const float * {  // or nullptr where there is none
                        if (t >= p.TDIM) return nullptr;
                        if (MODE == kGa) return tile * RT + r < p.RDIM ? p.gc + (size_t)(tile * RT + r) * N + n : nullptr;
                        const int2 px = pix_s[r];
                        const int oh = (px.y >> 16) + dh, ow = (px.y & 0xffff) + dw;
                        if (px.y < 0 || (unsigned)oh >= (unsigned)p.px.Ho || (unsigned)ow >= (unsigned)p.px.Wo) return nullptr;
                        return p.gc + (long)(px.x + dh * p.px.Wo + dw) * N + n;
                    };
                    if (p.vec_g) {
#pragma unroll
                        for (int i = 0; i < GR * (CT / 4) / THREADS; ++i) {
                            const int r = tid / (CT / 4) + THREADS / (CT / 4) * i;
                            const float *src = src_of(r0 + r);
                            cp_async16_zfill(g_s + r * CT + (c ^ (r & 4)), src ? src : p.gc, src != nullptr);
                        }
                    } else {
#pragma unroll 8
                        for (int i = 0; i < GR * CT / THREADS; ++i) {
                            const int r = tid / CT + THREADS / CT * i;
                            const float *src = src_of(r0 + r);
                            g_s[r * CT + (c ^ (r & 4))] = src ? *src : 0.f;
                        }
                    }
                }
                cp_async_commit();
                cp_async_wait<0>();
                __syncthreads();
                if (GR == RT || (unsigned)(tid - r0) < (unsigned)GR) {
                    const int r = tid - r0;
                    // (adding -0 changes no value; it makes a pair the result of one 64-bit instruction)
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int c = 8 * (j ^ l7);
#pragma unroll
                        for (int v = 0; v < 2; ++v) {
                            float4 f;
                            if (MODE == kGw) {
                                const float *q = g_s + (c + 4 * v) * GR + r;
                                f = make_float4(q[0], q[GR], q[2 * GR], q[3 * GR]);
                            } else {
                                f = *reinterpret_cast<const float4 *>(g_s + r * CT + ((c + 4 * v) ^ (r & 4)));
                            }
                            g[4 * j + 2 * v] = add2(pack2(f.x, f.y), minus_zero);
                            g[4 * j + 2 * v + 1] = add2(pack2(f.z, f.w), minus_zero);
                        }
                    }
                }
            }

            // where the sums of this block go
            float *dst = out0;
            const uint32_t doff = two_level ? tid : ooff;
            size_t dstride = ostride;
            bool add = block > 0;
            if (two_level) {
                dst = tmp0;
                dstride = RT;
                add = block % kRowsRun != 0;
            }

            __syncthreads();  // every value has been read
            store_cols(0);
            if (tid == 0) {
                // fresh barriers for this block: phases restart at 0 (nobody is waiting or arriving here)
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    if (!first_block) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(bar_full + 8 * b) : "memory");
                    mbar_init(bar_full + 8 * b, C::WARPS);
                }
            }
            first_block = false;
            __syncthreads();
            // Unit u's slabs are built at the start of unit u - 1, after the wait for that one's own slabs, into the buffer of
            // unit u - 3.  A warp that has seen unit u - 1 complete knows that every warp has built it, and so has left unit
            // u - 3: one barrier per unit is enough, and its arrival is a whole unit ahead of the wait for it.
            constexpr int UNITS = KC / KU;
            static_assert(UNITS > 2, "the next stage is written two units before it is read");
            build(0, cc_s);
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_full);

            uint32_t buf = 0, next = 1, par = 0;  // buffers of this unit and of the one after, parity of this round
            int stage = 0;
            for (int ks = kbeg; ks < kend; ks += KC, stage ^= 1) {
                const bool more = ks + KC < kend;
                if (more) fetch_cols(t0, ks + KC);
                const uint8_t *cb_ = cc_s + stage * C::CC_STAGE + KU * CT;  // term codes of the unit after
#pragma unroll 1
                for (int k4 = 0; k4 < KC / 4; ++k4) {
                    const int kg = ks + 4 * k4;
                    if (kg >= kend) break;
                    const uint32_t rw = __byte_perm(__byte_perm(raw[0], raw[1], 0x0040), __byte_perm(raw[2], raw[3], 0x0040), 0x5410) & MASK4;
                    fetch_rows(kg + 4);
                    auto begin_unit = [&](int it) {
                        mbar_wait(bar_full + 8 * buf, par, 1 + buf, abort_word, p.error_word);
                        build(next * UB, cb_);  // (past the last k: a slab that nobody reads)
                        if (it == UNITS - 3 && more) store_cols(stage ^ 1);
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_full + 8 * next);
                        cb_ = it == UNITS - 2 ? cc_s + (stage ^ 1) * C::CC_STAGE : cb_ + KU * CT;
                    };
                    auto end_unit = [&]() {
                        if (next == 0) par ^= 1;
                        buf = next;
                        if (++next == NB) next = 0;
                    };
                    // dot product of the slab row at `base` (bits 4 - 6 of it select the lane's first chunk)
                    auto dot = [&](uint32_t base) -> float {
                        constexpr int PF = 2;  // slab reads in flight ahead of their use
                        uint32_t q[PF][4];
                        auto fetch = [&](int j) {
                            uint32_t *d = q[j % PF];
                            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                                         : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(base ^ (j << 4)));
                        };
#pragma unroll
                        for (int j = 0; j < PF; ++j) fetch(j);
                        f32x2 acc[2];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const uint32_t w[4] = {q[j % PF][0], q[j % PF][1], q[j % PF][2], q[j % PF][3]};
                            if (j + PF < 8) fetch(j + PF);
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const f32x2 e = entries2(w[i], bias);
                                acc[i % 2] = j == 0 && i < 2 ? mul2(e, g[i]) : fma2(e, g[4 * j + i], acc[i % 2]);
                            }
                        }
                        const float2 t = unpack2(add2(acc[0], acc[1]));
                        return t.x + t.y;
                    };
                    float v[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (i % KU == 0) begin_unit(KU == 4 ? k4 : 4 * k4 + i);
                        v[i] = dot(__dp4a(rw, (uint32_t)C::U_ROW << (8 * i), ul + buf * UB + i % KU * C::U_BYTES));
                        if (i % KU == KU - 1) end_unit();
                    }
                    // (all four sums at the end: between the reads their branches cost 4 % and more)
                    float *d = dst + doff;
                    if (add) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) put<true>(d + i * dstride, v[i] * factor, in && kg + i < kend);
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; ++i) put<false>(d + i * dstride, v[i] * factor, in && kg + i < kend);
                    }
                    dst += 4 * dstride;
                }
            }
            if (two_level && in && (block % kRowsRun == kRowsRun - 1 || block == nblocks - 1)) {
                // the run is complete (its sums are this thread's own)
                float *o = out0 + ooff;
                const float *t = tmp0 + tid;
#pragma unroll 4
                for (int k = kbeg; k < kend; ++k, o += ostride, t += RT) {
                    const float s = __ldcg(t);
                    if (block >= kRowsRun) atomicAdd(o, s);
                    else *o = s;
                }
            }
        }
    }
}

}  // namespace sr

static size_t rows_block_floats(const RowsPlan &plan, long rows, int K, bool direct) {
    return plan.groups > 1 || !direct ? ((size_t)plan.groups * K * rows + 3) & ~(size_t)3 : 0;
}
static bool rows_needs_runs(const RowsPlan &plan) { return plan.group_blocks > kRowsChain; }

size_t rows_scratch_bytes(const RowsPlan &plan, long rows, int K, bool direct, int num_sms) {
    return (rows_block_floats(plan, rows, K, direct) + (rows_needs_runs(plan) ? (size_t)num_sms * plan.piece_k * kRowsTile : 0)) * sizeof(float);
}

namespace {

template <int BITS, int MODE>
int launch_rows(sr::Args p, float *out, float *scratch, bool direct, int num_sms, cudaStream_t stream) {
    using C = sr::Cfg<BITS>;
    auto kern = sr::slab_grad_rows_kernel<BITS, MODE>;
    if (!cuda_ok(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM))) return LUTGEMM_E_CUDA;
    p.error_word = device_error_word();
    if (!p.error_word) return LUTGEMM_E_CUDA;
    const RowsPlan &pl = p.plan;
    p.tiles = (p.RDIM + C::RT - 1) / C::RT;
    p.direct = direct && pl.groups == 1;
    p.out = p.direct ? out : scratch;
    p.tmp = rows_needs_runs(pl) ? scratch + rows_block_floats(pl, p.RDIM, p.K, direct) : nullptr;
    const long units = rows_units(pl, p.RDIM, p.K);
    const int grid = (int)(units < num_sms ? units : num_sms);
    kern<<<grid, C::THREADS, C::SMEM, stream>>>(p);
    return launch_status();
}

template <int BITS>
int launch_gw(sr::Args p, float *gw, float *scratch, int num_sms, cudaStream_t stream) {
    const int rc = launch_rows<BITS, sr::kGw>(p, gw, scratch, true, num_sms, stream);
    if (rc != LUTGEMM_OK || p.plan.groups == 1) return rc;
    return slab_reduce_blocks(scratch, gw, p.K, p.RDIM, p.plan.groups, false, nullptr, nullptr, kGradFactor, num_sms, stream);
}
template <int BITS>
int launch_ga(sr::Args p, float *ga, float *scratch, int num_sms, cudaStream_t stream) {
    const int rc = launch_rows<BITS, sr::kGa>(p, ga, scratch, false, num_sms, stream);
    if (rc != LUTGEMM_OK) return rc;
    return slab_reduce_blocks(scratch, ga, p.K, p.RDIM, p.plan.groups, true, nullptr, nullptr, kGradFactor, num_sms, stream);
}
template <int BITS>
int launch_gx(sr::Args p, float *gx, float *scratch, int num_sms, cudaStream_t stream) {
    const int rc = launch_rows<BITS, sr::kGx>(p, gx, scratch, true, num_sms, stream);
    if (rc != LUTGEMM_OK || p.plan.groups == 1) return rc;
    return slab_reduce_blocks(scratch, gx, p.K, p.RDIM, p.plan.groups, false, nullptr, &p.px, kGradFactor, num_sms, stream);
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

int backward_gw_rows(const float *gc, const uint8_t *w, float *gw, const int16_t *lut_gw, int bits, int M, int K, int N,
                     const RowsPlan &plan, float *scratch, const uint8_t *at, int at_pitch, int num_sms, cudaStream_t stream) {
    sr::Args p{};
    p.rows = w; p.row_stride = N; p.cols = at; p.col_pitch = at_pitch; p.lut = lut_gw; p.gc = gc;
    p.M = M; p.K = K; p.N = N; p.RDIM = N; p.TDIM = M; p.plan = plan;
    p.vec_c = 1;  // (the copy is 16-byte aligned, its pitch a multiple of 16)
    p.vec_g = N % 4 == 0 && aligned16(gc);
    switch (bits) {
        case 4: return launch_gw<4>(p, gw, scratch, num_sms, stream);
        case 6: return launch_gw<6>(p, gw, scratch, num_sms, stream);
        case 7: return launch_gw<7>(p, gw, scratch, num_sms, stream);
        case 8: return launch_gw<8>(p, gw, scratch, num_sms, stream);
    }
    return LUTGEMM_E_BITS;
}

int backward_ga_rows(const float *gc, const uint8_t *w, float *ga, const int16_t *lut_ga, int bits, int M, int K, int N,
                     const RowsPlan &plan, float *scratch, const uint8_t *at, int at_pitch, int num_sms, cudaStream_t stream) {
    sr::Args p{};
    p.rows = at; p.row_stride = at_pitch; p.cols = w; p.col_pitch = N; p.lut = lut_ga; p.gc = gc;
    p.M = M; p.K = K; p.N = N; p.RDIM = M; p.TDIM = N; p.plan = plan;
    p.vec_c = N % 16 == 0 && aligned16(w);
    p.vec_g = N % 4 == 0 && aligned16(gc);
    switch (bits) {
        case 4: return launch_ga<4>(p, ga, scratch, num_sms, stream);
        case 6: return launch_ga<6>(p, ga, scratch, num_sms, stream);
        case 7: return launch_ga<7>(p, ga, scratch, num_sms, stream);
        case 8: return launch_ga<8>(p, ga, scratch, num_sms, stream);
    }
    return LUTGEMM_E_BITS;
}

int backward_gx_rows(const float *gy, const uint8_t *x, const uint8_t *wmat, float *gx, const int16_t *lut_ga, int bits,
                     int Cout, const PixelClass &px, float *scratch, int num_sms, cudaStream_t stream) {
    sr::Args p{};
    p.rows = x; p.row_stride = (long)px.H * px.W; p.cols = wmat; p.lut = lut_ga; p.gc = gy;
    p.M = px.P; p.K = px.C; p.N = Cout; p.RDIM = px.P; p.TDIM = px.ntaps * Cout; p.px = px;
    p.plan = plan_rows(p.RDIM, p.TDIM, p.K, num_sms);
    p.vec_c = Cout % 16 == 0 && aligned16(wmat);
    p.vec_g = Cout % 4 == 0 && aligned16(gy);
    switch (bits) {
        case 4: return launch_gx<4>(p, gx, scratch, num_sms, stream);
        case 6: return launch_gx<6>(p, gx, scratch, num_sms, stream);
        case 7: return launch_gx<7>(p, gx, scratch, num_sms, stream);
        case 8: return launch_gx<8>(p, gx, scratch, num_sms, stream);
    }
    return LUTGEMM_E_BITS;
}

}  // namespace lutgemm
