// Forward LUT-GEMM for sm_100a, two output rows per thread: tiles of 1024 rows x 32 columns.
//     c[m,n] = sum_k LUT[a[m,k]][w[k,n]]        exact uint32 accumulate
//
// Per pair of k a slab is gathered once: for every activation code x a 128-byte row with LUT[x][w[k,n]] for the tile's 32 columns
// of the first k and then of the second (lutgemm_rows.cuh).  A thread owns rows 2t and 2t + 1 of the tile and reads the slab
// rows of their codes in 16-byte chunks.  Lane l takes chunk j ^ (l & 7), so that the eight lanes of a quarter-warp are on
// different bank quads whatever their codes are: lanes 4 - 7 start with the second k, and the accumulators of a lane hold its
// columns in the order (j ^ l) & 3.  Both k of a pair meet in one accumulator: S += w + v for the whole words, and the
// high halves H += w >> 16, v >> 16; sum(lo) = S - (H << 16), sum(hi) = H (mod 2^32).
//
// What bounds it: the shared-memory pipe, one wavefront per clock.  A slab row of 32 columns is built once per 1024 rows, half as
// often as by the kernel with a slab row of 64 columns per 512 rows (lutgemm_slab.cu).  Per k and 32768 look-ups 512 wavefronts
// of reads and 2^b of build; 4096^3: 8 bits 9.29 -> 6.05 ms (840 clocks per k and tile), 7 bits 6.74 -> 4.94 (685), 6 bits 6.54 -> 4.65,
// 4 bits 6.48 -> 4.48 (620); 262144 x 576 x 64 at 7 bits 1.09 -> 0.85 ms.
// Slab buffers change hands through one mbarrier per unit: see lutgemm_slab_rows.cu.  The activation codes come from
// the transposed copy at[k][m], 16 bits (both rows) per k.
// 512 threads leave a thread 128 registers: 4 and 6 bits spill 48 and 52 bytes, 7 and 8 bits none.
// Tiles and cut K as in lutgemm_slab.cu: whole tiles where they fill the persistent grid's waves, otherwise every CTA takes an
// equal contiguous share of all (tile, four k) units, and the parts of a tile that is cut are combined with integer atomics,
// which are exact in any order.  The sums leave through shared memory, so that rows are stored as whole 128-byte lines, with the layer's
// de-quantisation on the way where asked for.
// Replaces ApproxGemmForwardKernel, self_ops/src/approx_gemm_forward.cu:37-229.
#include "lutgemm_common.cuh"
#include "lutgemm_kernels.h"
#include "lutgemm_rows.cuh"
#include "lutgemm_waits.cuh"

namespace lutgemm {
namespace fr {

template <int BITS>
struct Cfg {
    using T = RowsTable<BITS>;
    static constexpr int Q = 1 << BITS;
    static constexpr int WARPS = 16, THREADS = 512, RT = kFwdRowsTile, CT = kFwdRowsCols;
    static constexpr int KC = 16;                         // k per operand stage
    static constexpr int KU = BITS == 8 ? 2 : 4, NB = 3;  // k per unit (two per slab), buffers
    static constexpr int SLABS = KU / 2, UB = SLABS * T::U_BYTES;
    static constexpr int CC_STAGE = KC * CT;
    static constexpr int OUT_BYTES = RT / 2 * CT * 4;     // sums of half of the rows on their way out
    static constexpr int U_AREA = NB * UB > OUT_BYTES ? NB * UB : OUT_BYTES;
    static constexpr int OFF_U = T::BYTES;
    static constexpr int OFF_CC = OFF_U + U_AREA;
    static constexpr int OFF_BAR = OFF_CC + 2 * CC_STAGE;
    static constexpr int SMEM = OFF_BAR + NB * 8 + 8;     // an mbarrier per buffer, abort word
    static_assert(OFF_U % 128 == 0 && T::TURN_BYTES <= U_AREA, "slab rows on fixed bank quads; the table passes through the buffers");
    static_assert(SMEM <= 232448, "shared memory budget");
};

struct Args {
    const uint8_t *at;  // [K][at_pitch], codes cut to the bit-width
    const uint8_t *w;   // [K][N]
    const uint16_t *lut;
    uint32_t *c;        // [M][N]
    int M, K, N, at_pitch;
    int tiles_c;
    long tiles;
    int share;          // 1: equal shares of (tile, four k) units per CTA, cut tiles combined with atomics; 0: whole tiles
    int vec_w;
    LayerEpilogue epi;  // epi.out != nullptr: the de-quantised fp32 layer output is stored instead of c
    int *error_word;    // device error word of the bounded waits
};

template <int BITS>
__global__ void __launch_bounds__(512, 1) forward_rows_kernel(const Args p) {
    using C = Cfg<BITS>;
    using T = RowsTable<BITS>;
    constexpr int RT = C::RT, CT = C::CT, KC = C::KC, KU = C::KU, NB = C::NB, UB = C::UB, UNITS = KC / KU;
    constexpr uint32_t MASK4 = (C::Q - 1) * 0x01010101u;
    const int M = p.M, K = p.K, N = p.N;

    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t *cc_s = smem + C::OFF_CC;
    const uint32_t u_addr = smem_u32(smem + C::OFF_U);
    const uint32_t bar_full = smem_u32(smem + C::OFF_BAR);
    volatile int *abort_word = reinterpret_cast<volatile int *>(smem + C::OFF_BAR + 8 * NB);
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5, l7 = lane & 7;

    stage_table_turned<BITS>(smem, smem + C::OFF_U, p.lut, 0u, tid);
    if (tid == 0) *abort_word = 0;
    if (tid < 2 * C::CC_STAGE / 16) reinterpret_cast<uint4 *>(cc_s)[tid] = make_uint4(0, 0, 0, 0);  // (codes past the last k)

    // ---- column codes: 16 k x 32 columns per stage, one 16-byte vector for each thread of warp 0 --------------------------------
    uint4 pcc = make_uint4(0, 0, 0, 0);
    auto fetch_cols = [&](int n0, int kbase) {
        if (tid < KC * CT / 16) {
            const int k = kbase + tid / (CT / 16), n = n0 + tid % (CT / 16) * 16;
            pcc = make_uint4(0, 0, 0, 0);
            if (k < K && n < N) {
                const uint8_t *src = p.w + (size_t)k * N + n;
                if (p.vec_w) {
                    pcc = *reinterpret_cast<const uint4 *>(src);
                } else {
                    uint32_t t[4] = {0, 0, 0, 0};
#pragma unroll
                    for (int q = 0; q < 16; ++q)
                        if (n + q < N) t[q >> 2] |= (uint32_t)src[q] << (8 * (q & 3));
                    pcc = make_uint4(t[0], t[1], t[2], t[3]);
                }
            }
        }
    };
    auto store_cols = [&](int stage) {
        if (tid < KC * CT / 16)
            *reinterpret_cast<uint4 *>(cc_s + stage * C::CC_STAGE + tid * 16) =
                make_uint4(pcc.x & MASK4, pcc.y & MASK4, pcc.z & MASK4, pcc.w & MASK4);
    };
    const SlabBuild<BITS> builder(smem_u32(smem), u_addr, tid);  // (a unit is one step at every bit-width)
    const uint32_t ul = u_addr + (l7 << 4);
    // dot-product weights: slab row of the k that the lane reads first, and of the other, for row 0 (row 1: one byte on)
    const uint32_t sel_first = (uint32_t)T::U_ROW << (l7 & 4 ? 16 : 0), sel_second = (uint32_t)T::U_ROW << (l7 & 4 ? 0 : 16);

    const int kunits = (K + 3) / 4;
    const long total = p.share ? p.tiles * kunits : p.tiles;
    long cur = p.share ? total * blockIdx.x / gridDim.x : (long)blockIdx.x;
    const long cur_end = p.share ? total * (blockIdx.x + 1) / gridDim.x : total;
    bool first = true;
    while (cur < cur_end) {
        int kbeg = 0, kend = K;
        long tile = cur;
        if (p.share) {
            tile = cur / kunits;
            const int k0 = (int)(cur - tile * kunits), nk = (int)min((long)(kunits - k0), cur_end - cur);
            kbeg = 4 * k0;
            kend = min(K, 4 * (k0 + nk));
            cur += nk;
        } else {
            cur += gridDim.x;
        }
        const bool partial = kbeg != 0 || kend != K;
        const int m0 = (int)(tile / p.tiles_c) * RT, n0 = (int)(tile % p.tiles_c) * CT;

        fetch_cols(n0, kbeg);
        // codes of both rows, two k at a time: raw[i] of k = kg + i, four k ahead of their use
        const uint8_t *rp = p.at + (size_t)kbeg * p.at_pitch;
        const uint32_t roff = min(m0 + 2 * tid, p.at_pitch - 2);  // (rows past M: any codes)
        uint32_t raw[4];
        auto fetch_rows = [&](int k) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                raw[i] = k + i < kend ? *reinterpret_cast<const uint16_t *>(rp + (size_t)i * p.at_pitch + roff) : 0u;
            rp += (size_t)4 * p.at_pitch;
        };
        fetch_rows(kbeg);

        // acc[r][4 j + w]: row r, word w (two columns) of chunk (j ^ l) & 3; [..][0] whole words, [..][1] high halves
        uint32_t acc[2][16][2];
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[r][i][0] = acc[r][i][1] = 0u;

        __syncthreads();  // the tile before (or the table staging) is done with every buffer
        store_cols(0);
        if (tid == 0) {
            // fresh barriers for this tile: phases restart at 0 (nobody is waiting or arriving here)
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                if (!first) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(bar_full + 8 * b) : "memory");
                mbar_init(bar_full + 8 * b, C::WARPS);
            }
        }
        first = false;
        __syncthreads();
        builder.step(0, cc_s);
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_full);

        uint32_t buf = 0, next = 1, par = 0;  // buffers of this unit and of the one after, parity of this round
        int stage = 0;
        for (int ks = kbeg; ks < kend; ks += KC, stage ^= 1) {
            const bool more = ks + KC < kend;
            if (more) fetch_cols(n0, ks + KC);
            const uint8_t *cb_ = cc_s + stage * C::CC_STAGE + KU * CT;  // column codes of the unit after
#pragma unroll 1
            for (int k4 = 0; k4 < KC / 4; ++k4) {
                const int kg = ks + 4 * k4;
                if (kg >= kend) break;
                const uint32_t rw[2] = {__byte_perm(raw[0], raw[1], 0x5410) & MASK4, __byte_perm(raw[2], raw[3], 0x5410) & MASK4};
                fetch_rows(kg + 4);
                // (see lutgemm_slab_rows.cu: the unit after is built into the buffer of two units ago)
                auto begin_unit = [&](int it) {
                    mbar_wait(bar_full + 8 * buf, par, 1 + buf, abort_word, p.error_word);
                    builder.step(next * UB, cb_);  // (past the last k: a slab that nobody reads)
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
                // the pair k, k + 1 from the slab at `ub`; with one k left the words of the other are left out
                auto use_pair = [&](uint32_t codes, uint32_t ub, bool both) {
                    const uint32_t keep_first = both || !(l7 & 4) ? ~0u : 0u, keep_second = both || (l7 & 4) ? ~0u : 0u;
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const uint32_t b0 = __dp4a(codes, sel_first << (8 * r), ub), b1 = __dp4a(codes, sel_second << (8 * r), ub ^ 64u);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            uint32_t w[4], v[4];
                            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                                         : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(b0 ^ (j << 4)));
                            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                                         : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(b1 ^ (j << 4)));
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                if (!both) {
                                    w[i] &= keep_first;
                                    v[i] &= keep_second;
                                }
                                acc[r][4 * j + i][0] += w[i] + v[i];
                                acc[r][4 * j + i][1] += w[i] >> 16;
                                acc[r][4 * j + i][1] += v[i] >> 16;
                            }
                        }
                    }
                };
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int k = kg + 2 * h;
                    if (KU == 2 && k >= kend) break;
                    if (KU == 2 || h == 0) begin_unit(KU == 2 ? 2 * k4 + h : k4);
                    const uint32_t ub = ul + buf * UB + (KU == 2 ? 0 : h * T::U_BYTES);
                    if (k + 1 < kend) use_pair(rw[h], ub, true);
                    else if (k < kend) use_pair(rw[h], ub, false);
                    if (KU == 2 || h == 1) end_unit();
                }
            }
        }

        // ---- sums out, rows of one parity at a time: [t][32 columns], the 16-byte pieces of threads 4 - 7 of eight swapped in
        //      pairs against bank conflicts; then a warp per row -----------------------------------------------------------
        uint32_t *out_s = reinterpret_cast<uint32_t *>(smem + C::OFF_U);
        LayerEpilogueScalars ev{};
        if (p.epi.out) ev = load_epilogue_scalars(p.epi);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            __syncthreads();  // every warp is done with the slabs, or with the rows of the other parity
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    uint32_t(&a)[2] = acc[r][4 * j + 2 * v], (&b)[2] = acc[r][4 * j + 2 * v + 1];
                    // low-half sum = whole-word sum - 65536 * high-half sum
                    *reinterpret_cast<uint4 *>(out_s + tid * CT + (((2 * ((j ^ l7) & 3) + v) ^ (l7 >> 2)) * 4)) =
                        make_uint4(a[0] - (a[1] << 16), a[1], b[0] - (b[1] << 16), b[1]);
                }
            __syncthreads();
            const int n = n0 + lane;
            if (n < N) {
#pragma unroll 4
                for (int i = 0; i < RT / 2 / C::WARPS; ++i) {
                    const int t = wp + C::WARPS * i, m = m0 + 2 * t + r;
                    if (m >= M) break;
                    const uint32_t sum = out_s[t * CT + (lane ^ (t & 4))];
                    if (p.epi.out) {
                        const int l = m % p.epi.L;
                        const float zw_box = __fmul_rn(ev.zw, p.epi.box[m]), zz_taps = __fmul_rn(ev.zz, p.epi.taps[l]);
                        p.epi.out[(size_t)m * N + n] = epilogue_value(p.epi, ev, sum, zw_box, zz_taps, l, n, N);
                    } else if (partial) {
                        atomicAdd(p.c + (size_t)m * N + n, sum);
                    } else {
                        p.c[(size_t)m * N + n] = sum;
                    }
                }
            }
        }
    }
}

}  // namespace fr

namespace {

template <int BITS>
int launch_forward_rows(fr::Args p, bool zeroed, int num_sms, cudaStream_t stream) {
    using C = fr::Cfg<BITS>;
    auto kern = fr::forward_rows_kernel<BITS>;
    if (!cuda_ok(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM))) return LUTGEMM_E_CUDA;
    p.error_word = device_error_word();
    if (!p.error_word) return LUTGEMM_E_CUDA;
    const long items = p.share ? p.tiles * ((p.K + 3) / 4) : p.tiles;
    const int grid = (int)(items < num_sms ? items : num_sms);
    if (p.share && !zeroed && !cuda_ok(cudaMemsetAsync(p.c, 0, (size_t)p.M * p.N * sizeof(uint32_t), stream))) return LUTGEMM_E_CUDA;
    kern<<<grid, C::THREADS, C::SMEM, stream>>>(p);
    return launch_status();
}

}  // namespace

int forward_rows(const uint8_t *w, uint32_t *c, const uint16_t *lut, int bits, int M, int K, int N, const uint8_t *at,
                 int at_pitch, const LayerEpilogue *epi, bool zeroed, int num_sms, cudaStream_t stream) {
    fr::Args p{};
    p.at = at; p.at_pitch = at_pitch; p.w = w; p.lut = lut; p.c = c; p.M = M; p.K = K; p.N = N;
    if (epi) p.epi = *epi;
    p.tiles_c = (N + kFwdRowsCols - 1) / kFwdRowsCols;
    p.tiles = (long)((M + kFwdRowsTile - 1) / kFwdRowsTile) * p.tiles_c;
    p.share = !epi && forward_rows_cut(M, K, N, num_sms);
    p.vec_w = N % 16 == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0;
    switch (bits) {
        case 4: return launch_forward_rows<4>(p, zeroed, num_sms, stream);
        case 6: return launch_forward_rows<6>(p, zeroed, num_sms, stream);
        case 7: return launch_forward_rows<7>(p, zeroed, num_sms, stream);
        case 8: return launch_forward_rows<8>(p, zeroed, num_sms, stream);
    }
    return LUTGEMM_E_BITS;
}

}  // namespace lutgemm
