// Quantisation prologue / de-quantisation epilogue of an approximate convolution layer, one pass each
// (the reference runs them as a dozen PyTorch elementwise kernels around its operator,
// micronet+/app_layers.py:147-181):
//
//   quantize:           codes[b,c,h,w] = clamp(rint(x / s_a - z_a), 0, qmax) as uint8, NCHW-contiguous, from
//                       an activation tensor of any dense layout (NCHW or channels-last), plus the channel
//                       sums chansum[b,h,w] = sum_c codes the zero-point cross term needs
//   epilogue:           out[m,co] = s_a s_w (y[m,co] + z_w box[m] + z_a sumw[l,co] + z_a z_w taps[l]) (+ bias[co])
//   quantize_backward:  gx = [0 <= rint(x / s_a - z_a) <= qmax] * s_w * (gcodes[b,c,h,w] + z_w boxT[b,h,w])
//                       written in the layout of x (straight-through rounding, clamp mask)
//
// Scales and zero points are read from device memory (they are module buffers refreshed every step), so
// no call synchronises with the host.
#include "lutgemm.h"
#include "lutgemm_codes.cuh"
#include "lutgemm_kernels.h"

namespace lutgemm {

namespace {

// Tile of 32 channels x 32 columns of one image row (b, h).  Reads follow the input's fastest dimension,
// writes follow w: for a channels-last input that is a transposition through shared memory.
template <bool BACKWARD>
__global__ void __launch_bounds__(256) quant_tile_kernel(const float *__restrict__ x, long sb, long sc, long sh, long sw,
                                                         int B, int C, int H, int W, const float *__restrict__ scale_p,
                                                         const float *__restrict__ zp_p, float qmax,
                                                         uint8_t *__restrict__ codes, float *__restrict__ chansum,
                                                         const float *__restrict__ gcodes, const float *__restrict__ boxT,
                                                         const float *__restrict__ sw_p, const float *__restrict__ zw_p,
                                                         float *__restrict__ gx) {
    __shared__ float tile[32][33];
    const Divisor scale = make_divisor(*scale_p);
    const float zp = *zp_p;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    const int ct = (C + 31) / 32;
    const bool chan_fast = sc == 1 && sw != 1;
    // one tile per CTA: blockIdx.x = (column tile, channel tile), blockIdx.y = image row, blockIdx.z = image (no
    // 64-bit divisions to decode a linear tile index: they cost more than the tile's arithmetic)
    {
        const int c0 = (int)(blockIdx.x % ct) * 32;
        const int w0 = (int)(blockIdx.x / ct) * 32;
        const int h = blockIdx.y, b = blockIdx.z;
        const float *xrow = x + b * sb + h * sh;
        // tile[c][w] = q (forward) or the clamp mask (backward)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int i = ty + 8 * r;
            const int c = chan_fast ? c0 + tx : c0 + i, w = chan_fast ? w0 + i : w0 + tx;
            float v = 0.f;
            if (c < C && w < W) {
                const float q = code_of(xrow[c * sc + w * sw], scale, zp);
                v = BACKWARD ? ((q >= 0.f && q <= qmax) ? 1.f : 0.f) : fminf(fmaxf(q, 0.f), qmax);
            }
            if (chan_fast) tile[tx][i] = v; else tile[i][tx] = v;
        }
        __syncthreads();
        if (!BACKWARD) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int c = c0 + ty + 8 * r, w = w0 + tx;
                if (c < C && w < W) codes[(((size_t)b * C + c) * H + h) * W + w] = (uint8_t)tile[ty + 8 * r][tx];
            }
            if (chansum && ty == 0 && w0 + tx < W) {
                float s = 0.f;
#pragma unroll 8
                for (int c = 0; c < 32; ++c) s += tile[c][tx];  // codes of channels >= C are 0
                atomicAdd(chansum + ((size_t)b * H + h) * W + w0 + tx, s);  // integer-valued sums < 2^24: exact in any order
            }
        } else {
            const float swt = *sw_p, zw = *zw_p;
            // g[c][w] = mask * s_w * (gcodes + z_w boxT), gathered along w, then written along x's fast dimension
            float gv[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int c = c0 + ty + 8 * r, w = w0 + tx;
                gv[r] = 0.f;
                if (c < C && w < W) {
                    float g = gcodes[(((size_t)b * C + c) * H + h) * W + w];
                    if (boxT) g = __fadd_rn(g, __fmul_rn(zw, boxT[((size_t)b * H + h) * W + w]));
                    gv[r] = tile[ty + 8 * r][tx] * __fmul_rn(swt, g);
                }
            }
            __syncthreads();
#pragma unroll
            for (int r = 0; r < 4; ++r) tile[ty + 8 * r][tx] = gv[r];
            __syncthreads();
            float *grow = gx + b * sb + h * sh;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int i = ty + 8 * r;
                const int c = chan_fast ? c0 + tx : c0 + i, w = chan_fast ? w0 + i : w0 + tx;
                if (c < C && w < W) grow[c * sc + w * sw] = chan_fast ? tile[tx][i] : tile[i][tx];
            }
        }
    }
}

// The same where input and output have the same layout and no channel sums or window terms come in (a linear layer): 16 values
// per thread.
template <bool BACKWARD>
__global__ void __launch_bounds__(256) quant_flat_kernel(const float *__restrict__ x, long n, const float *__restrict__ scale_p,
                                                         const float *__restrict__ zp_p, float qmax, uint8_t *__restrict__ codes,
                                                         const float *__restrict__ gcodes, const float *__restrict__ sw_p,
                                                         float *__restrict__ gx) {
    const Divisor scale = make_divisor(*scale_p);
    const float zp = *zp_p, swt = BACKWARD ? *sw_p : 0.f;
    constexpr int V = BACKWARD ? 8 : 16;
    for (long i = ((long)blockIdx.x * 256 + threadIdx.x) * V; i < n; i += (long)gridDim.x * 256 * V) {
        float4 f[V / 4], g[V / 4];
#pragma unroll
        for (int e = 0; e < V / 4; ++e) {
            f[e] = *reinterpret_cast<const float4 *>(x + i + 4 * e);
            if (BACKWARD) g[e] = *reinterpret_cast<const float4 *>(gcodes + i + 4 * e);
        }
        if (BACKWARD) {
#pragma unroll
            for (int e = 0; e < V / 4; ++e) {
                auto one = [&](float xv, float gv) {
                    const float q = code_of(xv, scale, zp);
                    return ((q >= 0.f && q <= qmax) ? 1.f : 0.f) * __fmul_rn(swt, gv);
                };
                *reinterpret_cast<float4 *>(gx + i + 4 * e) = make_float4(one(f[e].x, g[e].x), one(f[e].y, g[e].y), one(f[e].z, g[e].z), one(f[e].w, g[e].w));
            }
        } else {
            uint32_t w[V / 4];
#pragma unroll
            for (int e = 0; e < V / 4; ++e) {
                auto one = [&](float xv) { return (uint32_t)(uint8_t)fminf(fmaxf(code_of(xv, scale, zp), 0.f), qmax); };
                w[e] = one(f[e].x) | one(f[e].y) << 8 | one(f[e].z) << 16 | one(f[e].w) << 24;
            }
            *reinterpret_cast<uint4 *>(codes + i) = make_uint4(w[0], w[1 % (V / 4)], w[2 % (V / 4)], w[3 % (V / 4)]);
        }
    }
}

// The same for channels-last input, positions p = h * W + w in a row: tiles of 64 positions x 64 channels, 16-byte loads along the
// channels, four of them per thread in flight, turned in shared memory.  The tile of 32 x 32 in one image row with 4-byte
// accesses kept a third of the memory's bandwidth busy (64 x 256 x 56 x 56, forward 175 -> 55 us, backward 239 -> 110 us).
constexpr int kQP = 64, kQC = 64;
template <bool BACKWARD>
__global__ void __launch_bounds__(256) quant_nhwc_kernel(const float *__restrict__ x, int C, int P, const float *__restrict__ scale_p,
                                                         const float *__restrict__ zp_p, float qmax, uint8_t *__restrict__ codes,
                                                         float *__restrict__ chansum, const float *__restrict__ gcodes,
                                                         const float *__restrict__ boxT, const float *__restrict__ sw_p,
                                                         const float *__restrict__ zw_p, float *__restrict__ gx) {
    constexpr int BS = kQP + 4, GS = kQP + 1;  // bytes per channel of codes, floats per channel of gradients
    __shared__ __align__(16) uint8_t tile_s[BACKWARD ? kQC * GS * 4 : kQC * BS];
    const Divisor scale = make_divisor(*scale_p);
    const float zp = *zp_p;
    const int tid = threadIdx.x, cq = tid & 15, pg = tid >> 4;
    const int c0 = blockIdx.x * kQC, p0 = blockIdx.y * kQP, b = blockIdx.z;
    const int c = c0 + 4 * cq, p = p0 + 4 * pg;  // the thread's four channels and four positions
    const float *xb = x + ((size_t)b * P + p) * C + c;
    float4 f[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
        f[q] = c < C && p + q < P ? *reinterpret_cast<const float4 *>(xb + (size_t)q * C) : make_float4(0.f, 0.f, 0.f, 0.f);  // C % 4 == 0
    if (!BACKWARD) {
        uint32_t w[4] = {0u, 0u, 0u, 0u};  // codes of channel c + e, four positions
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float v[4] = {f[q].x, f[q].y, f[q].z, f[q].w};
            if (c < C && p + q < P)
#pragma unroll
                for (int e = 0; e < 4; ++e) w[e] |= (uint32_t)(uint8_t)fminf(fmaxf(code_of(v[e], scale, zp), 0.f), qmax) << (8 * q);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) *reinterpret_cast<uint32_t *>(tile_s + (4 * cq + e) * BS + 4 * pg) = w[e];
        if (chansum) {
            // sums over the tile's channels, two positions per word; 16 lanes hold the channels of four positions
            uint32_t even = 0u, odd = 0u;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                even += w[e] & 0x00ff00ffu;
                odd += (w[e] >> 8) & 0x00ff00ffu;
            }
#pragma unroll
            for (int d = 8; d; d >>= 1) {
                even += __shfl_xor_sync(0xffffffffu, even, d);
                odd += __shfl_xor_sync(0xffffffffu, odd, d);
            }
            if (cq < 4 && p + cq < P) {
                const uint32_t two = cq & 1 ? odd : even;
                atomicAdd(chansum + (size_t)b * P + p + cq, (float)(cq & 2 ? two >> 16 : two & 0xffffu));  // whole numbers below 2^24: exact in any order
            }
        }
        __syncthreads();
        // a channel's 64 positions by four threads, 16 bytes each
        const int oc = tid >> 2, op = (tid & 3) * 16;
        if (c0 + oc < C && p0 + op < P) {
            const uint32_t *src = reinterpret_cast<const uint32_t *>(tile_s + oc * BS + op);
            uint8_t *dst = codes + ((size_t)b * C + c0 + oc) * P + p0 + op;
            if (P % 16 == 0 && (reinterpret_cast<uintptr_t>(codes) & 15) == 0) {
                *reinterpret_cast<uint4 *>(dst) = make_uint4(src[0], src[1], src[2], src[3]);
            } else {
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    if (p0 + op + e < P) dst[e] = (uint8_t)(src[e >> 2] >> (8 * (e & 3)));
            }
        }
    } else {
        float *g_s = reinterpret_cast<float *>(tile_s);
        const float *gb = gcodes + ((size_t)b * C + c0) * P + p0;
        const bool vec = P % 4 == 0 && (reinterpret_cast<uintptr_t>(gcodes) & 15) == 0;
        float4 t[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {  // 16 channels per round, a channel's 64 positions by 16 threads
            const int ch = pg + 16 * r, pos = 4 * cq;
            t[r] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c0 + ch < C) {
                const float *src = gb + (size_t)ch * P + pos;
                if (vec) {
                    if (p0 + pos < P) t[r] = *reinterpret_cast<const float4 *>(src);
                } else {
                    if (p0 + pos < P) t[r].x = src[0];
                    if (p0 + pos + 1 < P) t[r].y = src[1];
                    if (p0 + pos + 2 < P) t[r].z = src[2];
                    if (p0 + pos + 3 < P) t[r].w = src[3];
                }
            }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float *d = g_s + (pg + 16 * r) * GS + 4 * cq;
            d[0] = t[r].x; d[1] = t[r].y; d[2] = t[r].z; d[3] = t[r].w;
        }
        __syncthreads();
        const float swt = *sw_p, zw = *zw_p;
        float *ob = gx + ((size_t)b * P + p) * C + c;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (c >= C || p + q >= P) break;
            const float v[4] = {f[q].x, f[q].y, f[q].z, f[q].w};
            const float window = boxT ? __fmul_rn(zw, boxT[(size_t)b * P + p + q]) : 0.f;
            float o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float code = code_of(v[e], scale, zp);
                float g = g_s[(4 * cq + e) * GS + 4 * pg + q];
                if (boxT) g = __fadd_rn(g, window);
                o[e] = ((code >= 0.f && code <= qmax) ? 1.f : 0.f) * __fmul_rn(swt, g);
            }
            *reinterpret_cast<float4 *>(ob + (size_t)q * C) = make_float4(o[0], o[1], o[2], o[3]);
        }
    }
}

// The whole prologue of a layer's forward pass in one launch: weight codes and their sums by the first `weight_blocks` blocks, the codes
// of channels-last activations and their channel sums by the others.  A block goes over all channels of 64 positions, the
// next 64 on their way meanwhile, so that it stores its channel sums and nobody has to zero and add to them.  Forward pass of
// ResNet-18, 16 images of 32 x 32: weight codes 184 us in all, activations 91 us, one after the other -> 185 us, three
// launches of the host's 5 us each -> one.
__global__ void __launch_bounds__(256) layer_prep_kernel(const WeightPrep wp, int weight_blocks, const float *__restrict__ x, int C, int P,
                                                         unsigned tiles_p, float qmax, uint8_t *__restrict__ codes,
                                                         float *__restrict__ chansum) {
    extern __shared__ uint32_t tap_sum[];
    if ((int)blockIdx.x < weight_blocks) {
        weight_prep_columns<8>(wp, blockIdx.x, tap_sum);
        return;
    }
    constexpr int BS = kQP + 4;
    __shared__ __align__(16) uint8_t tile_s[2][kQC * BS];
    const Divisor scale = make_divisor(wp.quant[0]);
    const float zp = wp.quant[1];
    const int tid = threadIdx.x, cq = tid & 15, pg = tid >> 4;
    const unsigned unit = blockIdx.x - weight_blocks, b = unit / tiles_p;
    const int p0 = (int)(unit - b * tiles_p) * kQP, p = p0 + 4 * pg;
    const float *xb = x + ((size_t)b * P + p) * C;
    const int oc = tid >> 2, op = (tid & 3) * 16;
    const bool wide = P % 16 == 0 && (reinterpret_cast<uintptr_t>(codes) & 15) == 0;
    float4 f[4];
    auto load = [&](int c) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
            f[q] = c < C && p + q < P ? *reinterpret_cast<const float4 *>(xb + (size_t)q * C + c) : make_float4(0.f, 0.f, 0.f, 0.f);  // C % 4 == 0
    };
    load(4 * cq);
    uint32_t total = 0u;  // of position p + cq, in the lanes with cq < 4
    int buf = 0;
    for (int c0 = 0; c0 < C; c0 += kQC, buf ^= 1) {
        const int c = c0 + 4 * cq;
        uint32_t w[4] = {0u, 0u, 0u, 0u};  // codes of channel c + e, four positions
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float v[4] = {f[q].x, f[q].y, f[q].z, f[q].w};
            if (c < C && p + q < P)
#pragma unroll
                for (int e = 0; e < 4; ++e) w[e] |= (uint32_t)(uint8_t)fminf(fmaxf(code_of(v[e], scale, zp), 0.f), qmax) << (8 * q);
        }
        if (c0 + kQC < C) load(c + kQC);
#pragma unroll
        for (int e = 0; e < 4; ++e) *reinterpret_cast<uint32_t *>(tile_s[buf] + (4 * cq + e) * BS + 4 * pg) = w[e];
        uint32_t even = 0u, odd = 0u;  // two positions per word
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            even += w[e] & 0x00ff00ffu;
            odd += (w[e] >> 8) & 0x00ff00ffu;
        }
#pragma unroll
        for (int d = 8; d; d >>= 1) {
            even += __shfl_xor_sync(0xffffffffu, even, d);
            odd += __shfl_xor_sync(0xffffffffu, odd, d);
        }
        const uint32_t two = cq & 1 ? odd : even;
        total += cq & 2 ? two >> 16 : two & 0xffffu;
        __syncthreads();  // (the other buffer was read before the barrier of this round)
        if (c0 + oc < C && p0 + op < P) {
            const uint32_t *src = reinterpret_cast<const uint32_t *>(tile_s[buf] + oc * BS + op);
            uint8_t *dst = codes + ((size_t)b * C + c0 + oc) * P + p0 + op;
            if (wide) {
                *reinterpret_cast<uint4 *>(dst) = make_uint4(src[0], src[1], src[2], src[3]);
            } else {
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    if (p0 + op + e < P) dst[e] = (uint8_t)(src[e >> 2] >> (8 * (e & 3)));
            }
        }
    }
    if (cq < 4 && p + cq < P) chansum[(size_t)b * P + p + cq] = (float)total;
}

// VEC: Cout is a multiple of 4 and the rows are 16-byte aligned, four channels per thread; otherwise a warp per output row m, lanes
// over the output channels (a row's terms and its position l = m mod L are computed once, nothing divides by Cout per value)
template <bool VEC>
__global__ void __launch_bounds__(256) conv_epilogue_kernel(const uint32_t *__restrict__ y, const float *__restrict__ box,
                                                            const float *__restrict__ sumw_t, const float *__restrict__ taps,
                                                            const float *__restrict__ sa_p, const float *__restrict__ sw_p,
                                                            const float *__restrict__ za_p, const float *__restrict__ zw_p,
                                                            const float *__restrict__ bias, float *__restrict__ out, long M,
                                                            int L, int Cout) {
    const float s = *sa_p * *sw_p, za = *za_p, zw = *zw_p, zz = za * zw;
    // separately rounded products and sums, in the order the PyTorch expression evaluates them
    auto one = [&](uint32_t sum, float zw_box, float sumw, float zz_taps, int co) {
        float acc = __fadd_rn((float)sum, zw_box);
        acc = __fadd_rn(acc, __fmul_rn(za, sumw));
        acc = __fadd_rn(acc, zz_taps);
        float o = __fmul_rn(s, acc);
        if (bias) o = __fadd_rn(o, bias[co]);
        return o;
    };
    if (VEC) {
        const int quads = Cout / 4;
        const long count = M * quads;
        for (long i = (long)blockIdx.x * 256 + threadIdx.x; i < count; i += (long)gridDim.x * 256) {
            const long m = count < (1L << 32) ? (unsigned)i / (unsigned)quads : i / quads;
            const int co = 4 * (int)(i - m * quads), l = (int)((unsigned)m % (unsigned)L);  // (M < 2^31)
            const uint4 v = reinterpret_cast<const uint4 *>(y)[i];
            const float4 sw = *reinterpret_cast<const float4 *>(sumw_t + (size_t)l * Cout + co);
            const float zw_box = __fmul_rn(zw, box[m]), zz_taps = __fmul_rn(zz, taps[l]);
            reinterpret_cast<float4 *>(out)[i] = make_float4(one(v.x, zw_box, sw.x, zz_taps, co), one(v.y, zw_box, sw.y, zz_taps, co + 1),
                                                             one(v.z, zw_box, sw.z, zz_taps, co + 2), one(v.w, zw_box, sw.w, zz_taps, co + 3));
        }
        return;
    }
    const int lane = threadIdx.x & 31, wrow = threadIdx.x >> 5;
    for (long m = (long)blockIdx.x * 8 + wrow; m < M; m += (long)gridDim.x * 8) {
        const int l = (int)(m % L);
        const float zw_box = __fmul_rn(zw, box[m]), zz_taps = __fmul_rn(zz, taps[l]);
        for (int co = lane; co < Cout; co += 32)
            out[m * Cout + co] = one(y[m * Cout + co], zw_box, sumw_t[(size_t)l * Cout + co], zz_taps, co);
    }
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
bool same_layout(long sb, long sc, long sh, long sw, int C, int H, int W) {  // NCHW
    return sw == 1 && sh == W && sc == (long)H * W && sb == (long)C * H * W;
}
bool channels_last(long sb, long sc, long sh, long sw, int C, int H, int W) {
    return sc == 1 && sw == C && sh == (long)W * C && sb == (long)H * W * C && C % 4 == 0;
}

}  // namespace

int quantize_codes(const float *x, long sb, long sc, long sh, long sw, int B, int C, int H, int W, const float *scale,
                   const float *zp_neg, float qmax, uint8_t *codes, float *chansum, int num_sms, cudaStream_t stream) {
    if (H > 65535 || B > 65535) return LUTGEMM_E_TOOLARGE;
    const long n = (long)B * C * H * W, P = (long)H * W;
    if (!chansum && same_layout(sb, sc, sh, sw, C, H, W) && n % 16 == 0 && aligned16(x) && aligned16(codes)) {
        const long blocks = (n / 16 + 255) / 256;
        quant_flat_kernel<false><<<(int)(blocks < 16L * num_sms ? blocks : 16L * num_sms), 256, 0, stream>>>(x, n, scale, zp_neg, qmax, codes, nullptr, nullptr, nullptr);
        return launch_status();
    }
    if (channels_last(sb, sc, sh, sw, C, H, W) && aligned16(x) && (P + kQP - 1) / kQP <= 65535) {
        const dim3 grid((unsigned)((C + kQC - 1) / kQC), (unsigned)((P + kQP - 1) / kQP), (unsigned)B);
        quant_nhwc_kernel<false><<<grid, 256, 0, stream>>>(x, C, (int)P, scale, zp_neg, qmax, codes, chansum, nullptr, nullptr, nullptr, nullptr, nullptr);
        return launch_status();
    }
    const dim3 grid((unsigned)(((W + 31) / 32) * ((C + 31) / 32)), (unsigned)H, (unsigned)B);
    quant_tile_kernel<false><<<grid, 256, 0, stream>>>(x, sb, sc, sh, sw, B, C, H, W, scale, zp_neg, qmax, codes, chansum,
                                                       nullptr, nullptr, nullptr, nullptr, nullptr);
    return launch_status();
}

int layer_prep(const float *x, long sb, long sc, long sh, long sw, int B, int C, int H, int W, float a_qmax, const float *weight,
               long s_co, long s_c, long s_h, long s_w, int Cout, int kh, int kw, float w_qmax, const float *quant, uint8_t *codes,
               float *chansum, uint8_t *wmat, float *wsum, int num_sms, cudaStream_t stream) {
    const int T = kh * kw;
    const long P = (long)H * W, tiles_p = (P + kQP - 1) / kQP, units = tiles_p * B;
    const int split = weight_prep_split(s_c, s_w, T);
    const long weight_blocks = (long)((Cout + 7) / 8) * (split ? T : 1);
    // One block for all channels where that leaves no more than eight rounds or the GPU full of blocks (16 x 512 x 4 x 4: 16 blocks of
    // eight rounds, hidden behind the weights); otherwise, and in other layouts, one launch each.
    if (T <= 512 && channels_last(sb, sc, sh, sw, C, H, W) && aligned16(x) && (C <= 8 * kQC || units >= num_sms) &&
        units + weight_blocks < (1L << 31)) {
        const WeightPrep w{weight, s_co, s_c, s_h, s_w, Cout, C, kh, kw, quant, w_qmax, wmat, wsum,
                           Cout % 8 == 0 && (reinterpret_cast<uintptr_t>(wmat) & 7) == 0, split};
        layer_prep_kernel<<<(unsigned)(units + weight_blocks), 256, 8 * T * sizeof(uint32_t), stream>>>(
            w, (int)weight_blocks, x, C, (int)P, (unsigned)tiles_p, a_qmax, codes, chansum);
        return launch_status();
    }
    // (the quantisation kernels add their channel tiles to the channel sums)
    if (!cuda_ok(cudaMemsetAsync(chansum, 0, (size_t)B * P * sizeof(float), stream))) return LUTGEMM_E_CUDA;
    const int rc = quantize_codes(x, sb, sc, sh, sw, B, C, H, W, quant, quant + 1, a_qmax, codes, chansum, num_sms, stream);
    if (rc != LUTGEMM_OK) return rc;
    return layer_weight_prep(weight, s_co, s_c, s_h, s_w, Cout, C, kh, kw, quant, w_qmax, wmat, wsum, stream);
}

int quantize_backward(const float *x, long sb, long sc, long sh, long sw, int B, int C, int H, int W, const float *scale,
                      const float *zp_neg, float qmax, const float *gcodes, const float *boxT, const float *s_w,
                      const float *z_w, float *gx, int num_sms, cudaStream_t stream) {
    if (H > 65535 || B > 65535) return LUTGEMM_E_TOOLARGE;
    const long n = (long)B * C * H * W, P = (long)H * W;
    if (!boxT && same_layout(sb, sc, sh, sw, C, H, W) && n % 8 == 0 && aligned16(x) && aligned16(gcodes) && aligned16(gx)) {
        const long blocks = (n / 8 + 255) / 256;
        quant_flat_kernel<true><<<(int)(blocks < 16L * num_sms ? blocks : 16L * num_sms), 256, 0, stream>>>(x, n, scale, zp_neg, qmax, nullptr, gcodes, s_w, gx);
        return launch_status();
    }
    if (channels_last(sb, sc, sh, sw, C, H, W) && aligned16(x) && aligned16(gx) && (P + kQP - 1) / kQP <= 65535) {
        const dim3 grid((unsigned)((C + kQC - 1) / kQC), (unsigned)((P + kQP - 1) / kQP), (unsigned)B);
        quant_nhwc_kernel<true><<<grid, 256, 0, stream>>>(x, C, (int)P, scale, zp_neg, qmax, nullptr, nullptr, gcodes, boxT, s_w, z_w, gx);
        return launch_status();
    }
    const dim3 grid((unsigned)(((W + 31) / 32) * ((C + 31) / 32)), (unsigned)H, (unsigned)B);
    quant_tile_kernel<true><<<grid, 256, 0, stream>>>(x, sb, sc, sh, sw, B, C, H, W, scale, zp_neg, qmax, nullptr, nullptr,
                                                      gcodes, boxT, s_w, z_w, gx);
    return launch_status();
}

int conv_epilogue(const uint32_t *y, const float *box, const float *sumw_t, const float *taps, const float *s_a,
                  const float *s_w, const float *z_a, const float *z_w, const float *bias, float *out, long M, int L,
                  int Cout, int num_sms, cudaStream_t stream) {
    const bool vec = Cout % 4 == 0 && M < (1L << 31) && aligned16(y) && aligned16(sumw_t) && aligned16(out);
    const long blocks = vec ? (M * (Cout / 4) + 255) / 256 : (M + 7) / 8, most = (vec ? 16L : 32L) * num_sms;
    auto kern = vec ? conv_epilogue_kernel<true> : conv_epilogue_kernel<false>;
    kern<<<(int)(blocks < most ? blocks : most), 256, 0, stream>>>(y, box, sumw_t, taps, s_a, s_w, z_a, z_w, bias, out, M, L, Cout);
    return launch_status();
}

}  // namespace lutgemm
