// Gradient LUT-GEMM kernels for sm_100a with a packed 16-bit "column-gathered slab" (512 x 64 tile).
//
//   grad_w:  gw[k,n] = 1/16 * sum_m T(a[m,k], w[k,n]) * gc[m,n]     rows r = m, columns c = n
//   grad_a:  ga[m,k] = 1/16 * sum_n gc[m,n] * T(a[m,k], w[k,n])     rows r = n, columns c = m
//   grad_x:  gx[b,c,h,w] = 1/16 * sum_{taps (i,j)} sum_n gy[m(b,h,w,i,j), n] * T(x[b,c,h,w], wmat[(c,i,j), n])
//            rows r = (tap, n), columns = input pixels, the k loop runs over the input channels c
//
// Per k a slab U_k[x][c] = T(x, cc[k,c]) is gathered once for all 2^b row codes x and the 64 columns of the tile, then
// every row reads slab row rc[r,k] contiguously (half a warp per row, four columns per lane in one 64-bit load,
// conflict-free by construction) and multiplies it with its grad_out entries, which stay in registers for the whole
// k loop.
//
// grad_x is the activation gradient of a convolution WITHOUT the unfolded intermediate: every tap that touches an input
// pixel sees the same activation code, so the sum over taps joins the sum over n in one long row dimension (kh*kw*Cout
// rows; the kernel exists with 576-row tiles for it as well), the column codes are the code image itself, the row codes are
// kh*kw rows of the weight matrix, and the result is written straight into the image gradient - no col2im, no atomics.  A
// strided convolution is cut into stride^2 classes of input pixels that each see a fixed subset of the taps.
//
// What bounds it: instruction issue (four per clock, packed fp32 instructions count twice) and the shared-memory pipe (one
// 128-byte wavefront per clock): 7 bits, grad_w of 4096 x 512 x 4096, per k and tile 3690 instructions, 1060 of them packed, and 980
// wavefronts in 1360 clocks; 8 bits 4860, 1335 and 1935.  The slab keeps the table's own 16 bits per entry, so a look-up costs half the
// wavefronts of an fp32 slab; the price is the conversion at each use.  It is done for two entries at a time: each 16-bit half goes, in
// offset-binary, behind the exponent of 2^23 (one byte permutation), one packed subtraction of 2^23 + 2^15 leaves the two signed entries
// exactly, and one packed multiply-add (fma.rn.f32x2) consumes them - 10 instructions per 128 look-ups of a warp
// against 8 with an fp32 slab, but 512 + build instead of 1024 + build wavefronts per 32768 look-ups.  Products and
// sums are the same fp32 operations as with an fp32 slab.
// 576-row tiles keep 72 registers of grad_out values and spill 4 to 16 bytes.
// With one barrier per unit and the staggered slab build of lutgemm_rows.cuh, against two barriers per unit and padded slab rows
// (grad_w, grad_a): 4096^3 at 7 bits 10.50, 11.12 -> 9.99, 10.09 ms, 6 bits 9.89, 10.71 -> 9.62, 9.63, 8 bits 15.19, 15.18 -> 14.15, 14.95;
// 262144 x 576 x 64 at 7 bits, grad_w 1.51 -> 1.46 ms.
//
// Hand-over between the warps of a CTA: at 7 bits and below three buffers of two slabs each and one mbarrier per buffer
// (lutgemm_slab_rows.cu); at 8 bits shared memory has room for two slabs, with a "full" and an "empty" mbarrier each, one arrival per
// warp (see lutgemm_slab_grad_tall.cu).  Every wait is bounded (lutgemm_waits.cuh).
// Partial sums: one per lane group, warp and k; one warp (rotating with k) adds the 32 of a column in four
// chains.
// A CTA takes the row blocks of a group one after the other and adds each to the group's sums in ascending order (the
// same thread stores and adds, so the reductions need no ordering between threads); groups are added by slab_reduce_blocks
// in ascending order: results are deterministic.  With one block of sums per row block the buffer grew with the rows: 0.82
// GB for the image gradient of a 3x3 layer of 256 channels at 56 x 56, batch 64, 7 bits, which now needs none.
// Replaces ApproxGemmBackwardKernelForGA / ForGB, self_ops/src/approx_gemm_backward.cu:13-258, 261-492, and for
// grad_x the unfold backward of self_ops/ops_py/approx_ops.py:556-571.
#include <type_traits>

#include "lutgemm_common.cuh"
#include "lutgemm_f32x2.cuh"
#include "lutgemm_kernels.h"
#include "lutgemm_rows.cuh"
#include "lutgemm_waits.cuh"

namespace lutgemm {
namespace sp {

enum { kGw = 1, kGa = 2, kGx = 3 };

template <int BITS, int RW_>
struct Cfg {
    static constexpr int Q = 1 << BITS;
    static constexpr int WARPS = 16, THREADS = 512, RW = RW_, RT = WARPS * RW, CT = 64;
    using T = RowsTable<BITS>;
    static constexpr int U_ROW = T::U_ROW;              // bytes per slab row
    static_assert(U_ROW == 2 * CT, "a slab row holds the tile's columns");
    static constexpr int KC = 16;                       // k per global fetch
    static constexpr int SC = BITS == 8 ? 8 : 16;       // k per shared-memory stage
    static constexpr int KP = BITS == 8 ? 1 : 2;        // slabs per buffer
    static constexpr int NB = BITS == 8 ? 2 : 3;        // buffers (shared memory has no room for a third at 8 bits)
    static constexpr int NSEG = RT / 16;                // 16-row code segments per k
    static constexpr int RC_LOADS = (KC * NSEG + THREADS - 1) / THREADS;
    static constexpr int TT_BYTES = T::BYTES, U_BYTES = T::U_BYTES;
    static constexpr int RC_STAGE = SC * RT, CC_STAGE = SC * CT;
    static constexpr int P_FLOATS = 2 * WARPS * CT;     // partial sums of one k: one row per half-warp
    static constexpr int OFF_U = TT_BYTES;
    static constexpr int OFF_RC = OFF_U + NB * KP * U_BYTES;
    static constexpr int OFF_CC = OFF_RC + 2 * RC_STAGE;
    static constexpr int OFF_PART = OFF_CC + 2 * CC_STAGE;
    static constexpr int OFF_PIX = OFF_PART + NB * KP * P_FLOATS * 4;  // (a set of sums per buffer)  grad_x: image offset of each column
    static constexpr int OFF_TAP = OFF_PIX + CT * 8;                  // grad_x: output offset {rows, columns} of each tap
    static constexpr int OFF_BAR = OFF_TAP + kMaxTaps * 8;
    static constexpr int SMEM = OFF_BAR + 2 * NB * 8 + 16;   // two mbarriers per buffer, abort word, work item
    static_assert(T::TURN_BYTES <= OFF_PART - OFF_U, "the table passes through the slab buffers and operand stages");
    static_assert(RW % 4 == 0 && RT % 16 == 0, "rows per warp");
    static_assert(U_BYTES % 16 == 0 && RC_STAGE % 16 == 0 && CC_STAGE % 16 == 0, "16-byte vectors");
    static_assert(SMEM <= 232448, "shared memory budget");
};

struct Args {
    const uint8_t *a;
    const uint8_t *w;
    const int16_t *lut;
    const float *gc;
    float *out;
    int M, K, N;               // kGx: M = pixels of the class (all images), K = channels, N = Cout
    int RDIM, CDIM;
    int tiles_r, tiles_c;
    int groups, group_blocks;  // row blocks are dealt to groups, each summed up by one CTA per column tile and k range
    int main_cells, tail_parts, tail_per;  // cells (group, column tile) with their whole K, and how K is cut for the others
    int direct;                // one group, and its sums go to their final place
    int vec_a, vec_w, vec_g;
    ConvGeom conv;
    int ga_scatter;     // grad_a of a convolution whose windows do not overlap: results go straight to the image
    const uint8_t *at;  // grad_w: transposed row codes at[k][m], rows at_pitch bytes apart
    int at_pitch;       // a multiple of 16; columns m >= M hold 0
    int *error_word;    // device error word of the bounded waits
    PixelClass px;      // kGx only
};

template <int BITS, int MODE, int RW>
__global__ void __launch_bounds__(512, 1) slab_grad_packed_kernel(const __grid_constant__ Args p) {
    using C = Cfg<BITS, RW>;
    constexpr int Q = C::Q, RT = C::RT, CT = C::CT, KC = C::KC, SC = C::SC, KP = C::KP, NB = C::NB;
    constexpr int WARPS = C::WARPS, THREADS = C::THREADS, NSEG = C::NSEG, RCL = C::RC_LOADS;
    constexpr int HALVES = KC / SC;  // shared-memory stages per fetched group of 16 k
    constexpr int NW = RW / 4;       // code words per warp; half h of the warp owns rows 4q + 2h and 4q + 2h + 1
    constexpr uint32_t MASK4 = (Q - 1) * 0x01010101u;

    const int M = p.M, K = p.K, N = p.N;
    const int RDIM = p.RDIM, CDIM = p.CDIM;

    extern __shared__ __align__(16) uint8_t smem[];
    uint8_t *rc_s = smem + C::OFF_RC;
    uint8_t *cc_s = smem + C::OFF_CC;
    float *part_s = reinterpret_cast<float *>(smem + C::OFF_PART);
    long long *pix_s = reinterpret_cast<long long *>(smem + C::OFF_PIX);
    int2 *tap_s = reinterpret_cast<int2 *>(smem + C::OFF_TAP);
    const uint32_t tt_addr = smem_u32(smem);
    const uint32_t u_addr = smem_u32(smem + C::OFF_U);
    const uint32_t bar_full = smem_u32(smem + C::OFF_BAR), bar_empty = bar_full + 8 * NB;
    volatile int *abort_word = reinterpret_cast<volatile int *>(smem + C::OFF_BAR + 16 * NB);
    int *work_s = reinterpret_cast<int *>(smem + C::OFF_BAR + 16 * NB + 4);  // grad_w, grad_a: cell and k range of the work item
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    const int half = lane >> 4, cq = lane & 15;  // half-warp and column quad (columns 4 cq .. 4 cq + 3)

    // ---- stage the gradient table in offset-binary; x = row code, y = column code, T(x,y) = lut[a*COL + w] -------
    // (grad_w: rows are activation codes, so the table is turned; grad_a / grad_x: rows are weight codes)
    const uint16_t *lut = reinterpret_cast<const uint16_t *>(p.lut);
    if (MODE == kGw) stage_table_turned<BITS>(smem, smem + C::OFF_U, lut, 0x80008000u, tid);
    else stage_table_plain<BITS>(smem, lut, 0x80008000u, tid);
    if (tid == 0) *abort_word = 0;
    __syncthreads();
    // (column codes past the last k: any codes, but codes)
    if (tid < 2 * C::CC_STAGE / 16) reinterpret_cast<uint4 *>(cc_s)[tid] = make_uint4(0, 0, 0, 0);
    if (MODE == kGx) {
        // pixel (hh, ww) of the class sits at h = ph + s hh; tap q connects it to output row (h - dh) / s = hh + eh
        for (int q = tid; q < p.px.ntaps; q += THREADS)
            tap_s[q] = make_int2((p.px.ph - p.px.dh[q]) / p.px.s, (p.px.pw - p.px.dw[q]) / p.px.s);
        __syncthreads();
    }

    // ---- operand staging: a group of 16 k is fetched into registers and written to shared memory SC k at a time:
    //      rc_s[stage][kk][r] (RT row codes per k), cc_s[stage][kk][c] (64 column codes per k) ---------------------
    uint4 prc[RCL], pcc = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int j = 0; j < RCL; ++j) prc[j] = make_uint4(0, 0, 0, 0);
    auto load16 = [&](const uint8_t *src, int valid) -> uint4 {  // up to 16 bytes, the rest 0
        uint32_t t[4] = {0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < 16; ++q)
            if (q < valid) t[q >> 2] |= (uint32_t)src[q] << (8 * (q & 3));
        return make_uint4(t[0], t[1], t[2], t[3]);
    };
    auto a_codes16 = [&](int m, int kbase) -> uint4 {  // a[m][kbase..kbase+15]
        m = min(m, M - 1);
        if (kbase >= K) return make_uint4(0, 0, 0, 0);
        if (p.conv.enabled) return conv_code16(p.a, p.conv, m, kbase, K);
        const uint8_t *src = p.a + (size_t)m * K + kbase;
        if (p.vec_a) return *reinterpret_cast<const uint4 *>(src);
        return load16(src, min(16, K - kbase));
    };
    auto w_codes16 = [&](int k, int n) -> uint4 {  // w[k][n..n+15]
        if (k >= K || n >= N) return make_uint4(0, 0, 0, 0);
        const uint8_t *src = p.w + (size_t)k * N + n;
        if (p.vec_w) return *reinterpret_cast<const uint4 *>(src);
        return load16(src, min(16, N - n));
    };
    // grad_x: row codes of channel k, rows r..r+15 with r = tap*N + n -> weight rows (k*T + t[tap])
    auto gx_row_codes16 = [&](int k, int r) -> uint4 {
        if (k >= K || r >= RDIM) return make_uint4(0, 0, 0, 0);
        int q = r / N, n = r - q * N;
        if (p.vec_w)  // N % 16 == 0: the 16 rows lie inside one tap
            return *reinterpret_cast<const uint4 *>(p.w + ((size_t)k * p.px.T + p.px.t[q]) * N + n);
        uint32_t t[4] = {0, 0, 0, 0};
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (r + i < RDIM) t[i >> 2] |= (uint32_t)p.w[((size_t)k * p.px.T + p.px.t[q]) * N + n] << (8 * (i & 3));
            if (++n == N) { n = 0; ++q; }
        }
        return make_uint4(t[0], t[1], t[2], t[3]);
    };
    // grad_x: the codes of pixel column tid % 64 in channels kbase + 2 (tid / 64) and + 1 (two byte loads per thread,
    // coalesced over the pixels)
    static_assert(MODE != kGx || THREADS * 2 == CT * KC, "two column codes per thread");
    auto gx_col_codes2 = [&](long long offset, bool valid, int kbase) -> uint32_t {
        const int k = kbase + 2 * (tid / CT);
        const size_t plane = (size_t)p.px.H * p.px.W;
        const uint8_t *src = p.a + offset + (size_t)k * plane;
        uint32_t t = 0;
        if (valid && k < K) t = src[0];
        if (valid && k + 1 < K) t |= (uint32_t)src[plane] << 8;
        return t;
    };
    auto fetch_group = [&](int r0, int c0, int group, bool first) {
        const int kbase = group * KC;
#pragma unroll
        for (int j = 0; j < RCL; ++j) {
            const int idx = tid + THREADS * j;  // (k, 16-row segment)
            const int gk = kbase + idx / NSEG, gr = r0 + (idx % NSEG) * 16;
            if ((KC * NSEG) % THREADS != 0 && idx >= KC * NSEG) prc[j] = make_uint4(0, 0, 0, 0);
            else if (MODE == kGw)
                prc[j] = (gk < K && gr < p.at_pitch) ? *reinterpret_cast<const uint4 *>(p.at + (size_t)gk * p.at_pitch + gr)
                                                     : make_uint4(0, 0, 0, 0);
            else prc[j] = MODE == kGx ? gx_row_codes16(gk, gr) : w_codes16(gk, gr);
        }
        if (MODE == kGx) {
            const int col = c0 + tid % CT;
            // (the first fetch of a tile is made before its table of image offsets is written)
            pcc.x = gx_col_codes2(first ? (long long)pixel_class_offset(p.px, min(col, CDIM - 1)) : pix_s[tid % CT], col < CDIM, kbase);
        } else if (tid < CT) {
            if (MODE == kGw) pcc = w_codes16(kbase + tid / (CT / 16), c0 + (tid % (CT / 16)) * 16);
            else pcc = a_codes16(c0 + tid, kbase);
        }
    };
    static_assert(KC * CT / 16 == CT, "column codes: one 16-byte vector for each of the first 64 threads");
    // writes the k range [hf*SC, hf*SC + SC) of the fetched group to `stage`, cut to BITS bits
    auto store_stage = [&](int stage, int hf) {
        uint8_t *rs = rc_s + stage * C::RC_STAGE;
        uint8_t *cs = cc_s + stage * C::CC_STAGE;
#pragma unroll
        for (int j = 0; j < RCL; ++j) {
            const int idx = tid + THREADS * j, kq = idx / NSEG;
            if (idx < KC * NSEG && (kq / SC == hf || HALVES == 1))
                *reinterpret_cast<uint4 *>(rs + (kq % SC) * RT + (idx % NSEG) * 16) =
                    make_uint4(prc[j].x & MASK4, prc[j].y & MASK4, prc[j].z & MASK4, prc[j].w & MASK4);
        }
        if (MODE == kGx) {
            const int k = 2 * (tid / CT);  // even, and SC is even: both codes go to the same stage
            if (k / SC == hf || HALVES == 1) {
                const uint32_t t = pcc.x & MASK4;
                cs[(k % SC) * CT + tid % CT] = (uint8_t)t;
                cs[(k % SC + 1) * CT + tid % CT] = (uint8_t)(t >> 8);
            }
        } else if (tid < CT) {
            const uint32_t tc[4] = {pcc.x & MASK4, pcc.y & MASK4, pcc.z & MASK4, pcc.w & MASK4};
            if (MODE == kGw) {
                const int kq = tid / (CT / 16);
                if (kq / SC == hf || HALVES == 1)
                    *reinterpret_cast<uint4 *>(cs + (kq % SC) * CT + (tid % (CT / 16)) * 16) = make_uint4(tc[0], tc[1], tc[2], tc[3]);
            } else {
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    if (q / SC == hf || HALVES == 1) cs[(q % SC) * CT + tid] = (uint8_t)(tc[q >> 2] >> (8 * (q & 3)));
            }
        }
    };
    const SlabBuild<BITS> builder(tt_addr, u_addr, tid);
    // add the 32 partial sums of one k in ascending order and store the tile's 64 columns (two per lane), or add them to
    // what this thread has stored for the row blocks before (reductions: nothing waits for the old value)
    auto reduce_store = [&](int k, const float *ps, float *obase, int c0, bool add) {
        // (four chains: their additions overlap, and their rounding errors are those of eight sums in a row)
        const f32x2 *p2 = reinterpret_cast<const f32x2 *>(ps) + lane;
        f32x2 c[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) c[i] = p2[i * (CT / 2)];
#pragma unroll
        for (int i = 4; i < 2 * WARPS; ++i) c[i & 3] = add2(c[i & 3], p2[i * (CT / 2)]);
        const f32x2 v = add2(add2(c[0], c[1]), add2(c[2], c[3]));
        float2 o = unpack2(v);
        if (p.direct) {  // (a power of two: the same sum whether it is scaled before or after)
            o.x *= kGradFactor;
            o.y *= kGradFactor;
        }
        const int col = c0 + 2 * lane;
        if (MODE != kGw && p.direct) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                if (col + e >= CDIM) break;
                const float ov = e ? o.y : o.x;
                if (MODE == kGx) {
                    float *dst = obase + (pix_s[2 * lane + e] + (long long)k * p.px.H * p.px.W);
                    if (add) atomicAdd(dst, ov);
                    else *dst = ov;
                } else if (p.ga_scatter) {
                    const long ix = conv_scatter_index(p.conv, col + e, k);
                    if (ix >= 0) obase[ix] = ov;
                } else {
                    obase[(size_t)(col + e) * K + k] = ov;
                }
            }
            return;
        }
        float *dst = obase + (size_t)k * CDIM + col;
        if (col + 1 < CDIM && (reinterpret_cast<uintptr_t>(dst) & 7) == 0) {
            if (add) atomicAdd(reinterpret_cast<float2 *>(dst), o);
            else *reinterpret_cast<float2 *>(dst) = o;
        } else if (add) {
            if (col < CDIM) atomicAdd(dst, o.x);
            if (col + 1 < CDIM) atomicAdd(dst + 1, o.y);
        } else {
            if (col < CDIM) dst[0] = o.x;
            if (col + 1 < CDIM) dst[1] = o.y;
        }
    };

    const f32x2 bias = pack2(-8421376.0f, -8421376.0f);  // -(2^23 + 2^15)
    const uint32_t wsel0 = (uint32_t)C::U_ROW << (16 * half), wsel1 = wsel0 << 8;  // dot-product weights of the lane's two rows

    const int items = p.main_cells + (p.groups * p.tiles_c - p.main_cells) * p.tail_parts;
    bool first_item = true;
    for (int item = blockIdx.x, block = 0; item < items;) {  // `block`: row block within the group
        int cell = item, kbeg = 0, kend = K;
        if (item >= p.main_cells) {
            const int j = item - p.main_cells;
            cell = p.main_cells + j / p.tail_parts;
            kbeg = (j % p.tail_parts) * p.tail_per;
            kend = min(K, kbeg + p.tail_per);
        }
        if constexpr (MODE != kGx) {
            // the compiler's schedule of the k loop depends on what it sees of these three: read back from shared memory
            // grad_w / grad_a take 10.00 / 10.09 ms for 4096^3 at 7 bits, straight from the branch 10.10 / 10.23 (grad_x: the other way
            // round, 6.81 against 6.93 ms at 8 bits for 16 x 256 x 56 x 56, 3x3)
            if (tid == 0) { work_s[0] = cell; work_s[1] = kbeg; work_s[2] = kend; }
            __syncthreads();
            cell = work_s[0];
            kbeg = work_s[1];
            kend = work_s[2];
        }
        const int group = cell / p.tiles_c, tc = cell % p.tiles_c;
        const int tr = group * p.group_blocks + block;
        const int r0 = tr * RT, c0 = tc * CT;
        const bool add = block > 0;

        // kbeg is a multiple of 16, so the first stage is half 0 of its group
        fetch_group(r0, c0, kbeg / KC, true);

        // (grad_x: the offsets of the taps come from a table and row -> (tap, n) is stepped, not divided: with four divisions
        // per load and the codes of a pixel's 16 channels read by one thread a tile of 64 channels spent a quarter of its time
        // here; 3x3, batch 256, 7 bits: 64 channels 2.17 -> 1.85 ms, 128 1.96 -> 1.75, 256 1.81 -> 1.65, 512 1.79 -> 1.64)
        // the grad_out block of this tile: g[2 (2q + j) + i] = entries of row 4q + 2h + j of the warp for the lane's
        // column pair i (columns 4 cq + 2 i, + 1)
        // (adding -0 changes no value; it makes the pair the result of one 64-bit instruction, so that it stays in an
        // aligned register pair - without it two moves per pair and k were spent on re-pairing the registers in grad_a)
        f32x2 g[RW];
        const f32x2 minus_zero = pack2(-0.0f, -0.0f);
        auto pair = [&](float lo, float hi) { return add2(pack2(lo, hi), minus_zero); };
        const int rb = r0 + wp * RW + 2 * half;  // row (q, j) of the lane is rb + 4 q + j
        const int cb = c0 + 4 * cq;
        if (MODE == kGw) {
#pragma unroll
            for (int q = 0; q < NW; ++q)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int m = rb + 4 * q + j;
                    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (m < M) {
                        const float *src = p.gc + (size_t)m * N + cb;
                        if (p.vec_g && cb < N) t = *reinterpret_cast<const float4 *>(src);  // N % 4 == 0
                        else {
                            if (cb < N) t.x = src[0];
                            if (cb + 1 < N) t.y = src[1];
                            if (cb + 2 < N) t.z = src[2];
                            if (cb + 3 < N) t.w = src[3];
                        }
                    }
                    g[2 * (2 * q + j)] = pair(t.x, t.y);
                    g[2 * (2 * q + j) + 1] = pair(t.z, t.w);
                }
        } else {
            // two rows (n, n + 1 of one output position) of four columns at a time
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float *base[2];          // grad_a: row of column e;  grad_x: position of tap offset 0
                int hh[2] = {0, 0}, ww[2] = {0, 0};
                bool valid[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int col = cb + 2 * i + e, cc = min(col, CDIM - 1);
                    valid[e] = col < CDIM;
                    if (MODE == kGa) {
                        base[e] = p.gc + (size_t)cc * N;
                    } else {
                        const int per = p.px.Hc * p.px.Wc, b = cc / per, rr = cc - b * per;
                        hh[e] = rr / p.px.Wc;
                        ww[e] = rr - hh[e] * p.px.Wc;
                        base[e] = p.gc + ((size_t)(b * p.px.Ho + hh[e]) * p.px.Wo + ww[e]) * N;
                    }
                }
                // &grad_out of (column e, row r = tap * N + n), or nullptr where there is none
                auto src_of = [&](int e, int r, int tap, int n) -> const float * {
                    if (!valid[e] || r >= RDIM) return nullptr;
                    if (MODE == kGa) return base[e] + r;
                    const int2 o = tap_s[tap];
                    if ((unsigned)(hh[e] + o.x) >= (unsigned)p.px.Ho || (unsigned)(ww[e] + o.y) >= (unsigned)p.px.Wo) return nullptr;
                    return base[e] + ((long)(o.x * p.px.Wo + o.y) * N + n);
                };
                int tap = MODE == kGx ? rb / N : 0, n = rb - tap * N;
#pragma unroll
                for (int q = 0; q < NW; ++q) {
                    const int r = rb + 4 * q;
                    float2 t[2];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        t[e] = make_float2(0.f, 0.f);
                        const float *src = src_of(e, r, tap, n);
                        if (p.vec_g) {  // N % 4 == 0: both rows share their tap and lie inside one 8-byte vector
                            if (src) t[e] = *reinterpret_cast<const float2 *>(src);
                        } else {
                            if (src) t[e].x = *src;
                            src = n + 1 < N || MODE == kGa ? src_of(e, r + 1, tap, n + 1) : src_of(e, r + 1, tap + 1, 0);
                            if (src) t[e].y = *src;
                        }
                    }
                    g[2 * (2 * q) + i] = pair(t[0].x, t[1].x);
                    g[2 * (2 * q + 1) + i] = pair(t[0].y, t[1].y);
                    if (MODE == kGx)
                        for (n += 4; n >= N; n -= N) ++tap;
                }
            }
        }

        __syncthreads();  // previous item (or the table staging) is done with every buffer
        store_stage((kbeg / SC) & 1, 0);
        if (MODE == kGx && tid < CT) pix_s[tid] = (long long)pixel_class_offset(p.px, min(c0 + tid, CDIM - 1));
        if (tid == 0) {
            // fresh barriers for this item: phases restart at 0 (nobody is waiting or arriving here)
#pragma unroll
            for (int b = 0; b < 2 * NB; ++b) {
                if (!first_item) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(bar_full + 8 * b) : "memory");
                mbar_init(bar_full + 8 * b, WARPS);
            }
        }
        first_item = false;
        __syncthreads();
        // unit u = KP consecutive k of one stage, in buffer u % NB; with NB buffers the slabs of unit u + NB - 1 are built
        // during unit u
        constexpr int UB = KP * C::U_BYTES;
        // one builder step: a slab at 8 bits, the two of a unit at fewer
        constexpr bool ONE_BARRIER = NB == 3;
        builder.step(0, cc_s + ((kbeg / SC) & 1) * C::CC_STAGE);
        __syncwarp();
        // the first unit is complete once every warp has arrived; with two buffers the second starts out released
        if (lane == 0) {
            mbar_arrive(bar_full);
            if (!ONE_BARRIER) mbar_arrive(bar_empty + 8);
        }

        float *obase = p.out + (p.direct ? (size_t)0 : (size_t)group * K * CDIM);

        const uint32_t uc = u_addr + cq * 8;
        f32x2 acc[2][2];  // [row parity j][column pair i]
        // rows of code words [QB, QE) of the warp: the lane's columns of the slab at `ua`, row codes of this k at `rbase`
        auto use_rows = [&](uint32_t ua, const uint8_t *rbase, auto qb_tag, auto qe_tag) {
            constexpr int QB = decltype(qb_tag)::value, QE = decltype(qe_tag)::value, NR = 2 * (QE - QB);
            // slab reads in flight ahead of their use (4096^3, grad_w / grad_a: 7 bits 10.03 / 10.08 ms with 2, 10.00 / 10.09 with 4, 10.08 /
            // 10.16 with 6, 10.14 / 10.31 with 8; 8 bits 14.62 / 14.96, 14.16 / 14.96, 14.95 / 14.96, 14.95 / 14.96)
            constexpr int PF = 4;
            uint32_t rv[QE - QB];
            if constexpr (RW % 16 == 0 && QB % 4 == 0 && QE % 4 == 0) {
#pragma unroll
                for (int q = 0; q < (QE - QB) / 4; ++q) {
                    const uint4 t = reinterpret_cast<const uint4 *>(rbase + QB * 4)[q];
                    rv[4 * q] = t.x; rv[4 * q + 1] = t.y; rv[4 * q + 2] = t.z; rv[4 * q + 3] = t.w;
                }
            } else if constexpr (RW % 8 == 0 && QB % 2 == 0 && QE % 2 == 0) {
#pragma unroll
                for (int q = 0; q < (QE - QB) / 2; ++q) {
                    const uint2 t = reinterpret_cast<const uint2 *>(rbase + QB * 4)[q];
                    rv[2 * q] = t.x; rv[2 * q + 1] = t.y;
                }
            } else {
#pragma unroll
                for (int q = 0; q < QE - QB; ++q) rv[q] = reinterpret_cast<const uint32_t *>(rbase + QB * 4)[q];
            }
            uint32_t w0[PF], w1[PF];
            auto fetch = [&](int i) {  // slab row address = base + 128 * code in one integer dot-product instruction
                asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(w0[i % PF]), "=r"(w1[i % PF])
                             : "r"(__dp4a(rv[i >> 1], i & 1 ? wsel1 : wsel0, ua)));
            };
#pragma unroll
            for (int i = 0; i < PF && i < NR; ++i) fetch(i);
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                const uint32_t a0 = w0[i % PF], a1 = w1[i % PF];
                if (i + PF < NR) fetch(i + PF);
                const int gi = 2 * (2 * QB + i);
                acc[i & 1][0] = fma2(entries2(a0, bias), g[gi], acc[i & 1][0]);
                acc[i & 1][1] = fma2(entries2(a1, bias), g[gi + 1], acc[i & 1][1]);
            }
        };
        using Q0 = std::integral_constant<int, 0>;
        using QH = std::integral_constant<int, RW == 24 ? 4 : NW / 2>;
        using QN = std::integral_constant<int, NW>;
        auto clear_acc = [&]() { acc[0][0] = acc[0][1] = acc[1][0] = acc[1][1] = pack2(0.f, 0.f); };
        // partial sums of one k: row 2 wp + h, the lane's four columns
        float *part_lane = part_s + (2 * wp + half) * CT + 4 * cq;
        auto store_part = [&](int slot) {
            const float2 lo = unpack2(add2(acc[0][0], acc[1][0])), hi = unpack2(add2(acc[0][1], acc[1][1]));
            *reinterpret_cast<float4 *>(part_lane + slot * C::P_FLOATS) = make_float4(lo.x, lo.y, hi.x, hi.y);
        };

        // Three buffers: unit u + 1 is built at the start of unit u into the buffer of unit u - 2, and one barrier per unit is
        // enough (lutgemm_slab_rows.cu); a warp that has seen unit u complete also knows that every warp has stored its
        // partial sums of unit u - 2, which are added up then.  Two buffers (8 bits): the build sits in the middle of the reads and waits
        // until every warp has released the unit before.
        constexpr int UNITS = SC / KP;  // per stage
        static_assert(UNITS > 2, "the next stage is written while no warp can still be reading it");
        uint32_t buf = 0, par = 0;  // buffer of this unit, parity of this round
        int stage = (kbeg / SC) & 1, hf = 0;
        for (int ks = kbeg; ks < kend; ks += SC, stage ^= 1, hf = HALVES == 1 ? 0 : hf ^ 1) {
            const bool more = ks + SC < kend;
            // the registers are free for the next group once the last stage of the current one is written
            if (more && (HALVES == 1 || hf == 1)) fetch_group(r0, c0, (ks + SC) / KC, false);
            const uint8_t *rb_ = rc_s + stage * C::RC_STAGE + wp * RW;
            const uint8_t *cb_ = cc_s + stage * C::CC_STAGE + KP * CT;  // column codes of the unit after
#pragma unroll 1
            for (int it = 0; it < UNITS; ++it) {
                const int k = ks + KP * it;
                if (k >= kend) break;
                const uint32_t next = buf == NB - 1 ? 0 : buf + 1;
                const uint32_t ua = uc + buf * UB;
                // the next stage is written before the full arrival of the unit during which its first slab is built
                const bool refill = it == UNITS - 3 && more;
                mbar_wait(bar_full + 8 * buf, par, 1 + buf, abort_word, p.error_word);  // the slabs of this unit are complete
                if constexpr (ONE_BARRIER) {
                    // (buffer and set of sums `next` belong to unit u - 2 as well)
                    if (k >= kbeg + 2 * KP && ((wp ^ (k - 2 * KP)) & (WARPS - KP)) == 0) {  // KP warps in turn
                        const int i = wp & (KP - 1);
                        reduce_store(k - 2 * KP + i, part_s + (next * KP + i) * C::P_FLOATS, obase, c0, add);
                    }
                    builder.step(next * UB, cb_);  // (past the last k: a slab that nobody reads)
                    if (refill) store_stage(stage ^ 1, HALVES == 1 ? 0 : hf ^ 1);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_full + 8 * next);
#pragma unroll
                    for (int i = 0; i < KP; ++i) {
                        if (i && k + i >= kend) break;
                        clear_acc();
                        use_rows(ua + i * C::U_BYTES, rb_ + i * RT, Q0{}, QN{});
                        store_part(buf * KP + i);
                    }
                } else {
                    clear_acc();
                    use_rows(ua, rb_, Q0{}, QH{});
                    // (same parity: the second buffer, which unit 0 waits for, starts out released)
                    mbar_wait(bar_empty + 8 * next, par, 1 + NB + next, abort_word, p.error_word);
                    if (k > kbeg && ((wp ^ (k - 1)) & (WARPS - 1)) == 0) reduce_store(k - 1, part_s + next * C::P_FLOATS, obase, c0, add);
                    if (k + 1 < kend) {
                        builder.step(next * UB, cb_);
                        if (refill) store_stage(stage ^ 1, HALVES == 1 ? 0 : hf ^ 1);
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_full + 8 * next);
                    }
                    use_rows(ua, rb_, QH{}, QN{});
                    store_part(buf);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_empty + 8 * buf);
                }
                rb_ += KP * RT;
                cb_ = it == UNITS - 2 ? cc_s + (stage ^ 1) * C::CC_STAGE : cb_ + KP * CT;
                if (next == 0) par ^= 1;
                buf = next;
            }
        }
        __syncthreads();  // every warp has stored its partial sums of the last units
        {
            // the last unit's, and with three buffers those of the one before it
            const int kl = kend - 1 - (kend - 1 - kbeg) % KP;  // first k of the last unit
            const int i = wp & (KP - 1);
#pragma unroll
            for (int back = ONE_BARRIER ? 1 : 0; back >= 0; --back) {
                const int ku = kl - back * KP;
                if (ku >= kbeg && ku + i < kend && ((wp ^ ku) & (WARPS - KP)) == 0)
                    reduce_store(ku + i, part_s + ((ku - kbeg) / KP % NB * KP + i) * C::P_FLOATS, obase, c0, add);
            }
        }
        if (++block == p.group_blocks || tr + 1 == p.tiles_r) {
            block = 0;
            item += gridDim.x;
        }
    }
}

}  // namespace sp

// Rows of a packed tile: the height that costs least over all row blocks, a k step of a tile taking about
// 78 + 5 rows-per-warp instructions per warp (slab build and loop, reads and arithmetic).  576 = 3 x 3 taps of 64 channels
// and half of 1152, 384 for row counts that would leave a quarter of 512 empty (7 bits, grad_a, 512-row tiles -> these:
// 12608 x 384 x 384 0.419 -> 0.359 ms, 12608 x 384 x 1152 1.244 -> 0.984 ms).
static int best_tile_rows(long rdim, bool with_384) {
    auto cost = [&](long rt, double step) { return (double)((rdim + rt - 1) / rt) * step; };
    int rt = 512;
    double c = cost(512, 1.0);
    if (cost(576, kPacked576Step) < c) { c = cost(576, kPacked576Step); rt = 576; }
    if (with_384 && cost(384, 0.83) < c) rt = 384;
    return rt;
}
int packed_ga_tile_rows(int N) { return best_tile_rows(N, true); }
int gx_tile_rows(long rdim) { return best_tile_rows(rdim, false); }

namespace {

template <int BITS, int MODE, int RW>
int launch_packed(sp::Args p, const PackedPlan &pp, float *out, float *scratch, int num_sms, cudaStream_t stream) {
    using C = sp::Cfg<BITS, RW>;
    auto kern = sp::slab_grad_packed_kernel<BITS, MODE, RW>;
    if (!cuda_ok(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM))) return LUTGEMM_E_CUDA;
    p.error_word = device_error_word();
    if (!p.error_word) return LUTGEMM_E_CUDA;
    p.tiles_r = (p.RDIM + C::RT - 1) / C::RT;
    p.tiles_c = (p.CDIM + C::CT - 1) / C::CT;
    p.groups = pp.groups;
    p.group_blocks = pp.group_blocks;
    // (grad_a is transposed on its way to its final place, by the reduction over the groups)
    p.direct = p.tiles_r == 1 || (MODE != sp::kGa && p.groups == 1);
    p.out = p.direct ? out : scratch;
    p.main_cells = pp.main_cells;
    p.tail_parts = pp.tail_parts;
    p.tail_per = pp.tail_per;
    const long items = pp.main_cells + ((long)p.groups * p.tiles_c - pp.main_cells) * pp.tail_parts;
    const int grid = (int)(items < num_sms ? items : num_sms);
    kern<<<grid, C::THREADS, C::SMEM, stream>>>(p);
    return launch_status();
}

template <int BITS, int MODE>
int launch_packed_gemm(const float *gc, const uint8_t *a, const uint8_t *w, float *out, const int16_t *lut, int M, int K,
                       int N, const ConvGeom &conv, const PackedPlan &plan, float *scratch, const uint8_t *at, int at_pitch,
                       int num_sms, cudaStream_t stream) {
    static_assert(sp::Cfg<BITS, 32>::RT == kSlabPackedRows, "tile height");
    sp::Args p{};
    p.a = a; p.w = w; p.lut = lut; p.gc = gc; p.M = M; p.K = K; p.N = N;
    p.RDIM = MODE == sp::kGa ? N : M;
    p.CDIM = MODE == sp::kGa ? M : N;
    p.conv = conv;
    p.at = at;
    p.at_pitch = at_pitch;
    p.ga_scatter = (MODE == sp::kGa && conv.enabled) ? 1 : 0;
    p.vec_a = !conv.enabled && (K % 16 == 0) && ((reinterpret_cast<uintptr_t>(a) & 15) == 0);
    p.vec_w = (N % 16 == 0) && ((reinterpret_cast<uintptr_t>(w) & 15) == 0);
    p.vec_g = (N % 4 == 0) && ((reinterpret_cast<uintptr_t>(gc) & 15) == 0);
    int rc, rt = kSlabPackedRows;
    if constexpr (MODE == sp::kGa) {
        rt = packed_ga_tile_rows(N);
        rc = rt == 384   ? launch_packed<BITS, MODE, 24>(p, plan, out, scratch, num_sms, stream)
             : rt == 576 ? launch_packed<BITS, MODE, 36>(p, plan, out, scratch, num_sms, stream)
                         : launch_packed<BITS, MODE, 32>(p, plan, out, scratch, num_sms, stream);
    } else {
        rc = launch_packed<BITS, MODE, 32>(p, plan, out, scratch, num_sms, stream);
    }
    if (rc != LUTGEMM_OK) return rc;
    if (MODE == sp::kGw ? plan.groups > 1 : p.RDIM > rt)
        return slab_reduce_blocks(scratch, out, K, p.CDIM, plan.groups, MODE == sp::kGa, p.ga_scatter ? &conv : nullptr, nullptr,
                                  kGradFactor, num_sms, stream);
    return LUTGEMM_OK;
}

template <int BITS>
int launch_packed_gx(const float *gy, const uint8_t *x, const uint8_t *wmat, float *gx, const int16_t *lut, int Cout,
                     const PixelClass &px, int B, float *scratch, int num_sms, cudaStream_t stream) {
    sp::Args p{};
    p.a = x; p.w = wmat; p.lut = lut; p.gc = gy;
    p.M = B * px.Hc * px.Wc; p.K = px.C; p.N = Cout;
    p.RDIM = px.ntaps * Cout;
    p.CDIM = p.M;
    p.px = px;
    p.vec_w = (Cout % 16 == 0) && ((reinterpret_cast<uintptr_t>(wmat) & 15) == 0);
    p.vec_g = (Cout % 4 == 0) && ((reinterpret_cast<uintptr_t>(gy) & 15) == 0);
    const int rw = gx_tile_rows(p.RDIM) / 16;
    const PackedPlan plan = plan_packed(p.RDIM, p.CDIM, p.K, 16 * rw, num_sms);
    const int rc = rw == 36 ? launch_packed<BITS, sp::kGx, 36>(p, plan, gx, scratch, num_sms, stream)
                            : launch_packed<BITS, sp::kGx, 32>(p, plan, gx, scratch, num_sms, stream);
    if (rc != LUTGEMM_OK) return rc;
    if (plan.groups > 1)
        return slab_reduce_blocks(scratch, gx, p.K, p.CDIM, plan.groups, false, nullptr, &px, kGradFactor, num_sms, stream);
    return LUTGEMM_OK;
}

}  // namespace

int backward_gw_slab_packed(const float *gc, const uint8_t *a, const uint8_t *w, float *gw, const int16_t *lut_gw,
                            int bits, int M, int K, int N, const ConvGeom &conv, const PackedPlan &plan, float *scratch,
                            const uint8_t *at, int at_pitch, int num_sms, cudaStream_t stream) {
    switch (bits) {
        case 4: return launch_packed_gemm<4, sp::kGw>(gc, a, w, gw, lut_gw, M, K, N, conv, plan, scratch, at, at_pitch, num_sms, stream);
        case 6: return launch_packed_gemm<6, sp::kGw>(gc, a, w, gw, lut_gw, M, K, N, conv, plan, scratch, at, at_pitch, num_sms, stream);
        case 7: return launch_packed_gemm<7, sp::kGw>(gc, a, w, gw, lut_gw, M, K, N, conv, plan, scratch, at, at_pitch, num_sms, stream);
        case 8: return launch_packed_gemm<8, sp::kGw>(gc, a, w, gw, lut_gw, M, K, N, conv, plan, scratch, at, at_pitch, num_sms, stream);
    }
    return LUTGEMM_E_BITS;
}

int backward_ga_slab_packed(const float *gc, const uint8_t *a, const uint8_t *w, float *ga, const int16_t *lut_ga,
                            int bits, int M, int K, int N, const ConvGeom &conv, const PackedPlan &plan, float *scratch,
                            int num_sms, cudaStream_t stream) {
    switch (bits) {
        case 4: return launch_packed_gemm<4, sp::kGa>(gc, a, w, ga, lut_ga, M, K, N, conv, plan, scratch, nullptr, 0, num_sms, stream);
        case 6: return launch_packed_gemm<6, sp::kGa>(gc, a, w, ga, lut_ga, M, K, N, conv, plan, scratch, nullptr, 0, num_sms, stream);
        case 7: return launch_packed_gemm<7, sp::kGa>(gc, a, w, ga, lut_ga, M, K, N, conv, plan, scratch, nullptr, 0, num_sms, stream);
        case 8: return launch_packed_gemm<8, sp::kGa>(gc, a, w, ga, lut_ga, M, K, N, conv, plan, scratch, nullptr, 0, num_sms, stream);
    }
    return LUTGEMM_E_BITS;
}

size_t gx_class_scratch_bytes(const PackedPlan &plan, const PixelClass &px) {
    return plan.groups > 1 ? (size_t)plan.groups * px.C * px.P * sizeof(float) : 0;
}

int backward_gx_class(const float *gy, const uint8_t *x, const uint8_t *wmat, float *gx, const int16_t *lut_ga, int bits,
                      int Cout, const PixelClass &px, int B, float *scratch, int num_sms, cudaStream_t stream) {
    switch (bits) {
        case 4: return launch_packed_gx<4>(gy, x, wmat, gx, lut_ga, Cout, px, B, scratch, num_sms, stream);
        case 6: return launch_packed_gx<6>(gy, x, wmat, gx, lut_ga, Cout, px, B, scratch, num_sms, stream);
        case 7: return launch_packed_gx<7>(gy, x, wmat, gx, lut_ga, Cout, px, B, scratch, num_sms, stream);
        case 8: return launch_packed_gx<8>(gy, x, wmat, gx, lut_ga, Cout, px, B, scratch, num_sms, stream);
    }
    return LUTGEMM_E_BITS;
}

// The blocks are added in 64 bits (these kernels wait for memory, the additions cost nothing) and rounded once: the rounding
// errors of many blocks in one fp32 chain showed (64 blocks of 64 terms: 1.8e-7 relative to the sums, now 1.0e-7).
struct Sum4 {
    double x, y, z, w;
    __device__ __forceinline__ float4 rounded() const { return make_float4((float)x, (float)y, (float)z, (float)w); }
};
__device__ __forceinline__ double sum_blocks(const float *p, size_t stride, int b0, int b1) {
    double s = 0.0;
#pragma unroll 4
    for (int b = b0; b < b1; ++b) s += p[b * stride];
    return s;
}
__device__ __forceinline__ Sum4 sum_blocks4(const float4 *p, size_t stride, int b0, int b1) {
    Sum4 s{0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
    for (int b = b0; b < b1; ++b) {
        const float4 v = p[b * stride];
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    return s;
}

// out[k][c] (TRANSPOSE=false) or out[c][k] (TRANSPOSE=true) = scale * sum_b part[b][k][c], b ascending.
// PLACE = 1: column c is an unfolded row m of a convolution with non-overlapping windows and (m,k) goes to its
// position in the image gradient (conv_scatter_index); PLACE = 2: column c is pixel c of a stride class and k a
// channel (pixel_class_offset).  Both with TRANSPOSE=false.
struct ReducePlace {
    ConvGeom conv;
    PixelClass px;
};
template <bool TRANSPOSE, int PLACE>
__global__ void slab_reduce_blocks_kernel(const float *__restrict__ part, float *__restrict__ out, int K, int C,
                                          int nblocks, float scale, const ReducePlace pl) {
    __shared__ float tile[32][33];
    const int tiles_c = (C + 31) / 32, tiles_k = (K + 31) / 32;
    const size_t KC_ = (size_t)K * C;
    for (int t = blockIdx.x; t < tiles_c * tiles_k; t += gridDim.x) {
        const int k0 = (t / tiles_c) * 32, c0 = (t % tiles_c) * 32;
        const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8 threads
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = k0 + ty + 8 * j, c = c0 + tx;
            float s = 0.f;
            if (k < K && c < C)
                s = (float)sum_blocks(part + (size_t)k * C + c, KC_, 0, nblocks);
            if (TRANSPOSE) tile[ty + 8 * j][tx] = s * scale;
            else if (k < K && c < C) {
                if (PLACE == 1) {
                    const long o = conv_scatter_index(pl.conv, c, k);
                    if (o >= 0) out[o] = s * scale;
                } else if (PLACE == 2) {
                    out[pixel_class_offset(pl.px, c) + (size_t)k * pl.px.H * pl.px.W] = s * scale;
                } else {
                    out[(size_t)k * C + c] = s * scale;
                }
            }
        }
        if (TRANSPOSE) {
            __syncthreads();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int c = c0 + ty + 8 * j, k = k0 + tx;
                if (k < K && c < C) out[(size_t)c * K + k] = tile[tx][ty + 8 * j];
            }
            __syncthreads();
        }
    }
}

// The same for plain outputs whose rows of partial sums are 16-byte aligned (C a multiple of 4): 16-byte loads, a
// 32 (k) x 128 (c) tile per step; the transposing form turns the tile in shared memory so that both sides stay
// coalesced.
template <bool TRANSPOSE>
__global__ void __launch_bounds__(256) slab_reduce_blocks_vec_kernel(const float *__restrict__ part, float *__restrict__ out,
                                                                     int K, int C, int nblocks, float scale) {
    __shared__ float tile[TRANSPOSE ? 32 * 129 : 1];
    const int tiles_c = (C + 127) / 128, tiles_k = (K + 31) / 32;
    const size_t KC_ = (size_t)K * C;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8 threads
    for (int t = blockIdx.x; t < tiles_c * tiles_k; t += gridDim.x) {
        const int k0 = (t / tiles_c) * 32, c0 = (t % tiles_c) * 128;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = k0 + ty + 8 * j, c = c0 + 4 * tx;
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k < K && c < C) {
                s = sum_blocks4(reinterpret_cast<const float4 *>(part + (size_t)k * C + c), KC_ / 4, 0, nblocks).rounded();
                s.x *= scale; s.y *= scale; s.z *= scale; s.w *= scale;
                if (!TRANSPOSE) *reinterpret_cast<float4 *>(out + (size_t)k * C + c) = s;
            }
            if (TRANSPOSE) {
                float *d = tile + (ty + 8 * j) * 129 + 4 * tx;
                d[0] = s.x; d[1] = s.y; d[2] = s.z; d[3] = s.w;
            }
        }
        if (TRANSPOSE) {
            __syncthreads();
            for (int cc = ty; cc < 128; cc += 8) {
                const int c = c0 + cc, k = k0 + tx;
                if (k < K && c < C) out[(size_t)c * K + k] = tile[tx * 129 + cc];
            }
            __syncthreads();
        }
    }
}

// Several blocks whose sums stay where they are: 32 vectors (or single sums, where blocks are not 16-byte aligned) per step
// of a CTA, the blocks shared out over its 16 warps in contiguous ranges.  One thread per sum and all blocks in a row left
// most of the GPU idle: 392 blocks of 64 x 256 sums took as long as a tenth of the kernel that made them, 16 blocks of
// 777 x 333 18 us.
template <bool VEC>
__global__ void __launch_bounds__(512) slab_reduce_many_kernel(const float *__restrict__ part, float *__restrict__ out,
                                                               long count, int nblocks, float scale) {
    __shared__ Sum4 sums[16][32];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int b0 = (int)((long)nblocks * ty / 16), b1 = (int)((long)nblocks * (ty + 1) / 16);
    for (long v0 = (long)blockIdx.x * 32; v0 < count; v0 += (long)gridDim.x * 32) {
        const long v = v0 + tx;
        Sum4 s{0.0, 0.0, 0.0, 0.0};
        if (v < count) {
            if (VEC) s = sum_blocks4(reinterpret_cast<const float4 *>(part) + v, count, b0, b1);
            else s.x = sum_blocks(part + v, count, b0, b1);
        }
        if (VEC) sums[ty][tx] = s;
        else sums[ty][tx].x = s.x;
        __syncthreads();
        if (ty == 0 && v < count) {
#pragma unroll
            for (int i = 1; i < 16; ++i) {
                s.x += sums[i][tx].x;
                if (VEC) { s.y += sums[i][tx].y; s.z += sums[i][tx].z; s.w += sums[i][tx].w; }
            }
            const float4 r = s.rounded();
            if (VEC) reinterpret_cast<float4 *>(out)[v] = make_float4(r.x * scale, r.y * scale, r.z * scale, r.w * scale);
            else out[v] = r.x * scale;
        }
        __syncthreads();
    }
}

int slab_reduce_blocks(const float *part, float *out, int K, int C, int nblocks, bool transpose, const ConvGeom *scatter,
                       const PixelClass *px, float scale, int num_sms, cudaStream_t stream) {
    if (!scatter && !px && !transpose && nblocks >= 4) {
        const bool vec = (long)K * C % 4 == 0 && (reinterpret_cast<uintptr_t>(part) & 15) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
        const long count = (long)K * C / (vec ? 4 : 1), ctas = (count + 31) / 32;
        const int grid = (int)(ctas < 4L * num_sms ? ctas : 4L * num_sms);
        if (vec) slab_reduce_many_kernel<true><<<grid, 512, 0, stream>>>(part, out, count, nblocks, scale);
        else slab_reduce_many_kernel<false><<<grid, 512, 0, stream>>>(part, out, count, nblocks, scale);
        return launch_status();
    }
    if (!scatter && !px && C % 4 == 0 && (reinterpret_cast<uintptr_t>(part) & 15) == 0 &&
        (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
        const long vtiles = (long)((K + 31) / 32) * ((C + 127) / 128);
        const int vgrid = (int)(vtiles < 8L * num_sms ? vtiles : 8L * num_sms);
        if (transpose) slab_reduce_blocks_vec_kernel<true><<<vgrid, 256, 0, stream>>>(part, out, K, C, nblocks, scale);
        else slab_reduce_blocks_vec_kernel<false><<<vgrid, 256, 0, stream>>>(part, out, K, C, nblocks, scale);
        return launch_status();
    }
    const long tiles = (long)((K + 31) / 32) * ((C + 31) / 32);
    const int rgrid = (int)(tiles < 8L * num_sms ? tiles : 8L * num_sms);
    ReducePlace pl{};
    if (scatter) {
        pl.conv = *scatter;
        slab_reduce_blocks_kernel<false, 1><<<rgrid, 256, 0, stream>>>(part, out, K, C, nblocks, scale, pl);
    } else if (px) {
        pl.px = *px;
        slab_reduce_blocks_kernel<false, 2><<<rgrid, 256, 0, stream>>>(part, out, K, C, nblocks, scale, pl);
    } else if (transpose) {
        slab_reduce_blocks_kernel<true, 0><<<rgrid, 256, 0, stream>>>(part, out, K, C, nblocks, scale, pl);
    } else {
        slab_reduce_blocks_kernel<false, 0><<<rgrid, 256, 0, stream>>>(part, out, K, C, nblocks, scale, pl);
    }
    return launch_status();
}

}  // namespace lutgemm
