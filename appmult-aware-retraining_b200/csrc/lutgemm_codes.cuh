// Codes of fp32 activations and weights: what the quantisation kernels and the weight kernels of a layer share.
#pragma once
#include "lutgemm_common.cuh"

namespace lutgemm {

__device__ __forceinline__ float code_of(float x, const Divisor &scale, float zp_neg) {
    return rintf(__fsub_rn(quotient(x, scale), zp_neg));  // two roundings, as x / scale - zp in PyTorch
}

struct WeightPrep {
    const float *weight;
    long s_co, s_c, s_h, s_w;
    int Cout, Cin, kh, kw;
    const float *quant;
    float qmax;
    uint8_t *wmat;
    float *wsum;
    int vec;    // eight channels in one store
    int split;  // a block per tap (weight_prep_split)
};
// Channels-last weights, whose input channels lie side by side, are cut by taps as well: their sums stay within a block.
__host__ __device__ inline bool weight_prep_split(long s_c, long s_w, int taps) { return s_c < s_w && taps > 1; }

// By block number `block`, CO output channels, one tap of them or all: codes of weight[co, :, :, :] (any strides) written as columns of
// wmat[K, Cout], K ordered (cin, kh, kw); wsum[co, t] = sum over cin of the codes of tap t.  A thread handles one k of all CO
// channels, so its reads are independent of each other and its codes leave in one CO-byte store; those of its next k are
// on their way meanwhile.  Threads follow the weights' own order (channels-last weights, one tap of them at a time, have the input
// channel innermost).  The sums are integers (exact in any order; shared-memory atomics are native for integers only), added up
// inside the warp first where there is one tap.  384 x 1536 linear layer: 44.7 us with one channel per block, byte stores and fp32 atomics -> 4.2 us.
// Channels-last 3x3 weights of ResNet-18, all layers and with their activations: 280 us with a block per eight channels, 185 us by taps.
template <int CO>
__device__ __forceinline__ void weight_prep_columns(const WeightPrep &w, int block, uint32_t *tap_sum) {
    const int groups = (w.Cout + CO - 1) / CO, co0 = block % groups * CO, T = w.kh * w.kw;
    const int t0 = w.split ? block / groups : 0, nt = w.split ? 1 : T;
    const int K = w.Cin * nt, lane = threadIdx.x & 31, threads = blockDim.x;
    const bool one_tap = nt == 1;
    const Divisor scale = make_divisor(w.quant[2]);
    const float zp = w.quant[3];
    for (int u = threadIdx.x; u < CO * nt; u += threads) tap_sum[u] = 0u;
    __syncthreads();
    int c = 0, t = t0;
    float x[CO];
    auto load = [&](int i) {
        c = one_tap ? i : i / T;
        t = one_tap ? t0 : i - c * T;
        const int row = t / w.kw, col = t - row * w.kw;
        const float *src = w.weight + co0 * w.s_co + c * w.s_c + row * w.s_h + col * w.s_w;
#pragma unroll
        for (int e = 0; e < CO; ++e) x[e] = co0 + e < w.Cout ? src[e * w.s_co] : 0.f;
    };
    if ((int)threadIdx.x < K) load(threadIdx.x);
    for (int i0 = 0; i0 < K; i0 += threads) {  // (whole warps: the sum over the warp below needs every lane)
        const int i = i0 + threadIdx.x, tap = t - t0;
        uint32_t q[CO];
#pragma unroll
        for (int e = 0; e < CO; ++e) q[e] = i < K ? (uint32_t)(uint8_t)fminf(fmaxf(code_of(x[e], scale, zp), 0.f), w.qmax) : 0u;
        uint8_t *dst = w.wmat + (size_t)(c * T + t) * w.Cout + co0;
        if (i + threads < K) load(i + threads);
        if (i < K) {
            if (CO == 8 && w.vec) {
                *reinterpret_cast<uint2 *>(dst) = make_uint2(q[0] | q[1 % CO] << 8 | q[2 % CO] << 16 | q[3 % CO] << 24,
                                                             q[4 % CO] | q[5 % CO] << 8 | q[6 % CO] << 16 | q[7 % CO] << 24);
            } else {
#pragma unroll
                for (int e = 0; e < CO; ++e)
                    if (co0 + e < w.Cout) dst[e] = (uint8_t)q[e];
            }
        }
        if (one_tap) {
#pragma unroll
            for (int e = 0; e < CO; ++e) {
                const uint32_t sum = __reduce_add_sync(0xffffffffu, q[e]);
                if (lane == 0) atomicAdd(&tap_sum[e], sum);  // (a warp behind the last k adds 0)
            }
        } else if (i < K) {
#pragma unroll
            for (int e = 0; e < CO; ++e) atomicAdd(&tap_sum[e * nt + tap], q[e]);
        }
    }
    __syncthreads();
    for (int u = threadIdx.x; u < CO * nt; u += threads)
        if (co0 + u / nt < w.Cout) w.wsum[(size_t)(co0 + u / nt) * T + t0 + u % nt] = (float)tap_sum[u];
}

}  // namespace lutgemm
