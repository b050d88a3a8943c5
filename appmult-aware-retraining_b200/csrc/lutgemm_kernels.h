// Internal launch interfaces between the C-ABI translation unit and the kernel translation units.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace lutgemm {

// Failure bookkeeping: the CUDA error behind a LUTGEMM_E_CUDA status is kept per host thread so that
// lutgemm_status_string can name it (cudaGetLastError clears the runtime's own record).
void record_cuda_error(cudaError_t e);
inline bool cuda_ok(cudaError_t e) {
    if (e == cudaSuccess) return true;
    record_cuda_error(e);
    return false;
}
// status of the launch just made on this thread
int launch_status();

// scratch of the weight gradient under the choice by fixed limits, or of the family that is forced (lutgemm_api.cu)
size_t base_gw_scratch_bytes(int bits, int M, int K, int N);

struct ConvGeom;    // lutgemm_common.cuh; geometry.enabled == 0 means `a` is a plain [M,K] matrix
struct PixelClass;  // lutgemm_common.cuh; the input pixels of one stride class of a convolution and their taps
struct LayerEpilogue;  // lutgemm_common.cuh; optional de-quantisation applied where the forward kernels store

// `epi` (optional): the kernel stores the de-quantised fp32 layer output epi->out instead of the uint32 sums c
int forward_rowbcast(const uint8_t *a, const uint8_t *w, uint32_t *c, const uint16_t *lut, int bits, int M, int K,
                     int N, const ConvGeom &conv, const LayerEpilogue *epi, int num_sms, cudaStream_t stream);

// `at` (optional): the activation codes transposed, at[k][m] with rows at_pitch bytes apart (transpose_codes); `zeroed`: c holds
// zeros already, which the parts of a cut K are added to
int forward_slab(const uint8_t *a, const uint8_t *w, uint32_t *c, const uint16_t *lut, int bits, int M, int K, int N,
                 const ConvGeom &conv, const uint8_t *at, int at_pitch, const LayerEpilogue *epi, bool zeroed, int num_sms,
                 cudaStream_t stream);

// forward kernel with two output rows per thread (lutgemm_forward_rows.cu), tiles of 1024 rows x 32 columns; `at` as above,
// not optional
constexpr int kFwdRowsTile = 1024, kFwdRowsCols = 32;
int forward_rows(const uint8_t *w, uint32_t *c, const uint16_t *lut, int bits, int M, int K, int N, const uint8_t *at,
                 int at_pitch, const LayerEpilogue *epi, bool zeroed, int num_sms, cudaStream_t stream);
// whether it cuts K where it is free to: whole tiles would leave the last wave of the persistent grid badly filled
inline bool forward_rows_cut(int M, int K, int N, int num_sms) {
    const long tiles = (long)((M + kFwdRowsTile - 1) / kFwdRowsTile) * ((N + kFwdRowsCols - 1) / kFwdRowsCols);
    const long waves = (tiles + num_sms - 1) / num_sms;
    // (a cut costs about as much as 24 k: two parts per CTA to zero and to combine)
    return (double)waves * K > (double)tiles * K / num_sms + 24;
}

// operand chunks of forward_slab by bulk-tensor copies (default) or by vector loads through registers
void slab_fwd_set_tma(bool on);
// number of K ranges forward_slab cuts a problem into when it is free to (1 = none; a fused epilogue needs 1)
int slab_fwd_ksplits(int M, int K, int N, int num_sms);

// How a slab kernel cuts K (outputs are per k, so the parts are independent work items): the number of parts and the k
// per part (a multiple of 16) for which a persistent grid of num_sms CTAs finishes first, when an item of `per` k costs
// per + item_overhead steps.  Up to 64 parts, so that few tiles still fill the GPU; beyond 16 items per CTA another part
// gains less than 1 / 16, and the search (a microsecond of host time per call) ends.
struct KSplit {
    int parts, per;
    long waves;
};
inline KSplit choose_ksplit(long tiles, int K, int num_sms, int item_overhead) {
    const unsigned chunks = (unsigned)(K + 15) / 16, sms = (unsigned)num_sms;
    KSplit best{1, (int)chunks * 16, (tiles + num_sms - 1) / num_sms};
    long cost = best.waves * (best.per + item_overhead);
    unsigned last = chunks;
    for (unsigned s = 2; s <= 64 && s <= chunks && tiles * s <= 16L * num_sms; ++s) {
        const unsigned per = (chunks + s - 1) / s;  // in chunks
        if (per == last) continue;                  // more parts of the same length: some would get no work
        last = per;
        const unsigned parts = (chunks + per - 1) / per, waves = ((unsigned)tiles * parts + sms - 1) / sms;
        const long c = (long)waves * (16 * per + item_overhead);
        if (c < cost) { cost = c; best = KSplit{(int)parts, (int)per * 16, (long)waves}; }
    }
    return best;
}
// in k steps: operand fetch, grad_out block (gathered in grad_a and grad_x), first slabs
constexpr int kPackedGwOverhead = 5, kPackedItemOverhead = 10, kTallItemOverhead = 4;

// rows of the reduction dimension per CTA tile of the packed-slab gradient kernels
constexpr int kSlabPackedRows = 512;
constexpr double kPacked576Step = 1.13;  // time of a k step with 576 rows
// How the packed gradient kernels deal out their work.  The row blocks of a column tile are cut into groups of
// group_blocks; one CTA adds up a group's blocks in turn, so a group needs one block of partial sums.  A cell is (group,
// column tile): the first main_cells of them, whole rounds of the persistent grid, are taken with their whole K, the
// others with K cut (outputs are per k) so that the last round is full too.
struct PackedPlan {
    int groups, group_blocks;
    int main_cells, tail_parts, tail_per;
    long steps, items;  // k steps of the CTA that has most to do, its item overheads among them, and its work items (row blocks each)
};
inline PackedPlan deal_cells(long groups, long blocks, long tiles_c, int K, int num_sms, int item_overhead) {
    const long cells = groups * tiles_c, rounds = cells / num_sms, tail = cells % num_sms;
    const int whole = (K + 15) / 16 * 16;
    PackedPlan p{(int)groups, (int)blocks, (int)(rounds * num_sms), 1, whole, rounds * (whole + item_overhead), rounds};
    if (tail) {
        const KSplit ks = choose_ksplit(tail, K, num_sms, item_overhead);
        p.tail_parts = ks.parts;
        p.tail_per = ks.per;
        p.steps += ks.waves * (ks.per + item_overhead);
        p.items += ks.waves;
    }
    p.steps *= blocks;
    p.items *= blocks;
    return p;
}
// Where the tiles fill the GPU anyway, the largest groups that cost no time: one block of sums per row block made the
// buffer grow with the rows (0.9 GB for grad_w and 0.8 GB for the image gradient of a 3x3 layer of 256 channels at
// 56 x 56, batch 64).  Fewer blocks of sums save their reading (4 bytes at 4000 per clock, a step is about 1500 clocks).
inline PackedPlan plan_packed(long rdim, long cdim, int K, int tile_rows, int num_sms, int item_overhead = kPackedItemOverhead,
                              long most_blocks = 1L << 30) {
    const long tiles_r = (rdim + tile_rows - 1) / tile_rows, tiles_c = (cdim + 63) / 64;
    const PackedPlan alone = deal_cells(tiles_r, 1, tiles_c, K, num_sms, item_overhead);
    if (tiles_r * tiles_c < num_sms) return alone;
    const unsigned sms = (unsigned)num_sms;
    const long whole = (K + 15) / 16 * 16 + item_overhead;
    for (long blocks = tiles_r < most_blocks ? tiles_r : most_blocks; blocks > 1; --blocks) {
        const long groups = (tiles_r + blocks - 1) / blocks;
        if ((tiles_r + groups - 1) / groups < blocks) continue;  // as many groups of fewer blocks
        const long most = alone.steps + alone.steps / 256 + (tiles_r - groups) * tiles_c * K / 23400;
        // (most candidates cannot do it even with an even last round: the search for their K split is left out)
        const long rounds = groups * tiles_c / sms, tail = groups * tiles_c % sms;
        if (blocks * (rounds * whole + (tail ? tail * K / sms + item_overhead : 0)) > most) continue;
        const PackedPlan p = deal_cells(groups, blocks, tiles_c, K, num_sms, item_overhead);
        if (p.steps <= most) return p;
    }
    return alone;
}
// (grad_w: at most 16 blocks in a chain of additions, so that a long sum is still added up in two levels)
inline PackedPlan plan_packed_gw(long M, long N, int K, int num_sms) {
    return plan_packed(M, N, K, kSlabPackedRows, num_sms, kPackedGwOverhead, 16);
}
int packed_ga_tile_rows(int N);  // grad_a: rows of its tile (384, 512 or 576)
// gradient slab kernels with 16-bit slab entries (converted where they are used)
// `at`: the row codes transposed, at[k][m] with rows at_pitch bytes apart (transpose_codes); `plan`: plan_packed_gw or, for
// grad_a, plan_packed of the problem
int backward_gw_slab_packed(const float *gc, const uint8_t *a, const uint8_t *w, float *gw, const int16_t *lut_gw,
                            int bits, int M, int K, int N, const ConvGeom &conv, const PackedPlan &plan, float *scratch,
                            const uint8_t *at, int at_pitch, int num_sms, cudaStream_t stream);
int backward_ga_slab_packed(const float *gc, const uint8_t *a, const uint8_t *w, float *ga, const int16_t *lut_ga,
                            int bits, int M, int K, int N, const ConvGeom &conv, const PackedPlan &plan, float *scratch,
                            int num_sms, cudaStream_t stream);
// fp32 slab entries and a tall tile (1024 rows x 32 columns)
constexpr int kSlabTallRows = 1024;
int slab_tall_row_blocks(int rdim);
// lut_f32 (optional, bits <= 7): the gradient table as fp32 in the same padded layout; it replaces the int16
// table and the 1/16 scale
int backward_gw_slab_tall(const float *gc, const uint8_t *a, const uint8_t *w, float *gw, const int16_t *lut_gw,
                          const float *lut_f32, int bits, int M, int K, int N, const ConvGeom &conv, float *scratch,
                          const uint8_t *at, int at_pitch, int num_sms, cudaStream_t stream);
int backward_ga_slab_tall(const float *gc, const uint8_t *a, const uint8_t *w, float *ga, const int16_t *lut_ga,
                          const float *lut_f32, int bits, int M, int K, int N, const ConvGeom &conv, float *scratch,
                          int num_sms, cudaStream_t stream);
// ---- gradient kernel with one thread per output row (lutgemm_slab_rows.cu): tiles of 512 rows x 64 terms ------------------
constexpr int kRowsTile = 512, kRowsTerms = 64;
constexpr int kRowsChain = 16, kRowsRun = 8;     // term blocks added in one chain; above it, length of the runs
constexpr int kRowsMaxPer = 128;                // k per work item where sums of runs are kept (bounds their buffer)
constexpr int kRowsBlockOverhead = 7;         // in k steps: grad_out block, first slabs
// How its work is dealt out.  The term blocks of a row tile are cut into groups of group_blocks; the cells (tile, group), each
// with its K in units of four k, are laid end to end and every CTA takes an equal share of the units: pieces of at most
// piece_k k of one cell, all term blocks of the group one after the other.
struct RowsPlan {
    int groups, group_blocks, piece_k;
    double steps, loads;  // k steps of one CTA, and how often it loads a block's grad_out values and fills its slabs
};
constexpr int kRowsUnit = 4;
inline long rows_units(const RowsPlan &p, long rows, int K) {
    return (rows + kRowsTile - 1) / kRowsTile * p.groups * ((K + kRowsUnit - 1) / kRowsUnit);
}
// units and blocks are counted in 32 bits
inline bool rows_supported(long rows, long terms, int K) {
    return (double)rows / kRowsTile * 128 * (K / kRowsUnit + 1) < 1e9 && terms < (1L << 31) - kRowsTerms && rows < (1L << 31) - kRowsTile;
}
// The number of groups that finishes first: more groups fill the GPU where tiles and K alone do not, and spread a block's
// grad_out loads over more k, at the price of another block of sums each.
inline RowsPlan plan_rows(long rows, long terms, int K, int num_sms) {
    const long tiles = (rows + kRowsTile - 1) / kRowsTile;
    const int blocks = (int)((terms + kRowsTerms - 1) / kRowsTerms), kp = (K + kRowsUnit - 1) / kRowsUnit * kRowsUnit;
    constexpr double kMostSums = 96e6;  // bytes of sums of several groups
    RowsPlan best{};
    double best_cost = 0;
    for (int g = 1; g <= blocks && g <= 128; g += g < 4 ? 1 : g < 16 ? 2 : g < 32 ? 4 : 16) {
        RowsPlan p{};
        p.group_blocks = (blocks + g - 1) / g;
        p.groups = (blocks + p.group_blocks - 1) / p.group_blocks;
        const double sums = p.groups > 1 ? 8.0 * p.groups * K * (double)rows / 4000 / 1200 + 5 : 0;
        if (best.groups && (sums >= best_cost || (double)p.groups * K * rows * sizeof(float) > kMostSums)) break;
        const long share = (rows_units(p, rows, K) + num_sms - 1) / num_sms * kRowsUnit;
        const int most = p.group_blocks > kRowsChain && kp > kRowsMaxPer ? kRowsMaxPer : kp;
        const long pieces = (share + most - 1) / most;
        p.piece_k = most == kp ? kp : (int)((share + pieces - 1) / pieces + kRowsUnit - 1) / kRowsUnit * kRowsUnit;
        // (a share begins and ends inside a cell: one piece more than its length asks for, where there is more than one cell)
        p.steps = (double)p.group_blocks * share;
        p.loads = p.group_blocks * ((double)pieces + (tiles * p.groups > 1));
        const double cost = p.steps + kRowsBlockOverhead * p.loads + sums;
        if (!best.groups || cost < best_cost) { best = p; best_cost = cost; }
    }
    return best;
}
// floats of its scratch buffer: blocks of sums where they do not go to their final place, and sums of runs
size_t rows_scratch_bytes(const RowsPlan &plan, long rows, int K, bool direct, int num_sms);
// `at`: the activation codes transposed, at[k][m] with rows at_pitch bytes apart (transpose_codes)
int backward_gw_rows(const float *gc, const uint8_t *w, float *gw, const int16_t *lut_gw, int bits, int M, int K, int N,
                     const RowsPlan &plan, float *scratch, const uint8_t *at, int at_pitch, int num_sms, cudaStream_t stream);
int backward_ga_rows(const float *gc, const uint8_t *w, float *ga, const int16_t *lut_ga, int bits, int M, int K, int N,
                     const RowsPlan &plan, float *scratch, const uint8_t *at, int at_pitch, int num_sms, cudaStream_t stream);
int backward_gx_rows(const float *gy, const uint8_t *x, const uint8_t *wmat, float *gx, const int16_t *lut_ga, int bits,
                     int Cout, const PixelClass &px, float *scratch, int num_sms, cudaStream_t stream);
// reads (and clears) the device-side error word of the bounded barrier waits; synchronises the device
int read_and_clear_device_error(int *value);
// launches a one-warp kernel whose barrier wait can never be satisfied (it must time out with error id 99)
int bounded_wait_selftest(cudaStream_t stream);
// out[k][c] (or out[c][k] when transpose) = 1/16 * sum over row blocks of part[b][k][c], b ascending; with
// `scatter` (columns are unfolded rows of that convolution) or `px` (columns are pixels of that class, k a
// channel) the sums go to their positions in the image gradient instead
int slab_reduce_blocks(const float *part, float *out, int K, int C, int nblocks, bool transpose, const ConvGeom *scatter,
                       const PixelClass *px, float scale, int num_sms, cudaStream_t stream);
// activation gradient of a convolution for the input pixels of one stride class, written into gx[B,C,H,W]
// (packed slab kernel in pixel mode: no unfolded gradient, no col2im); scratch: gx_class_scratch_bytes()
int gx_tile_rows(long rdim);  // rows of its tile for a class of rdim = taps * Cout rows
size_t gx_class_scratch_bytes(const PackedPlan &plan, const PixelClass &px);  // plan_packed of the class
int backward_gx_class(const float *gy, const uint8_t *x, const uint8_t *wmat, float *gx, const int16_t *lut_ga, int bits,
                      int Cout, const PixelClass &px, int B, float *scratch, int num_sms, cudaStream_t stream);
// the same with the column-broadcast gather kernel (whole table in shared memory, no slab) for `nclasses` stride
// classes at once (up to four per launch, so that small images still fill the GPU): better where the row dimension
// taps * Cout is too short to amortise a slab build
int backward_gx_bcast(const float *gy, const uint8_t *x, const uint8_t *wmat, float *gx, const int16_t *lut_ga, int bits,
                      int Cout, const PixelClass *classes, int nclasses, int num_sms, cudaStream_t stream);
// hand-over between the warps of the tall gradient kernels: per-buffer mbarriers (default) or one CTA barrier per k
void slab_tall_set_handover(bool on);


// at[k][m] = a[m][k] cut to `bits` bits (or the unfolded code image when conv.enabled); rows `pitch` bytes apart,
// pitch a multiple of 16 and >= M, columns m >= M are written as 0.  `zero` (optional): words to set to zero in the same launch.
int transpose_codes(const uint8_t *a, uint8_t *at, int M, int K, int pitch, const ConvGeom &conv, int bits,
                    uint32_t *zero, long zero_words, cudaStream_t stream);

// quantisation prologue / epilogue of an approximate convolution layer (lutgemm_quant.cu); strides in elements
int quantize_codes(const float *x, long sb, long sc, long sh, long sw, int B, int C, int H, int W, const float *scale,
                   const float *zp_neg, float qmax, uint8_t *codes, float *chansum, int num_sms, cudaStream_t stream);
// codes and channel sums of the activations, codes and tap sums of the weights of a layer; quant = {s_a, z_a, s_w, z_w}
int layer_prep(const float *x, long sb, long sc, long sh, long sw, int B, int C, int H, int W, float a_qmax, const float *weight,
               long s_co, long s_c, long s_h, long s_w, int Cout, int kh, int kw, float w_qmax, const float *quant, uint8_t *codes,
               float *chansum, uint8_t *wmat, float *wsum, int num_sms, cudaStream_t stream);
int quantize_backward(const float *x, long sb, long sc, long sh, long sw, int B, int C, int H, int W, const float *scale,
                      const float *zp_neg, float qmax, const float *gcodes, const float *boxT, const float *s_w,
                      const float *z_w, float *gx, int num_sms, cudaStream_t stream);
int conv_epilogue(const uint32_t *y, const float *box, const float *sumw_t, const float *taps, const float *s_a,
                  const float *s_w, const float *z_a, const float *z_w, const float *bias, float *out, long M, int L,
                  int Cout, int num_sms, cudaStream_t stream);

// small one-pass kernels of the layer wiring (lutgemm_layer_aux.cu); strides in elements, quant = {s_a, z_a, s_w, z_w}
int layer_update_ranges(const float *act_lo, const float *act_hi, const float *w_lo, const float *w_hi, float *act_min,
                        float *act_max, float *act_seen, float *w_min, float *w_max, float *w_seen, float keep,
                        float momentum, float a_qmax, float w_qmax, float eps, float *quant, cudaStream_t stream);
int layer_weight_prep(const float *weight, long s_co, long s_c, long s_h, long s_w, int Cout, int Cin, int kh, int kw,
                      const float *quant, float qmax, uint8_t *wmat, float *wsum, cudaStream_t stream);
int layer_cross_terms(const float *wsum, int Cout, const ConvGeom &g, float *sumw_t, float *taps, int num_sms,
                      cudaStream_t stream);
int layer_window_sum(const float *img, const ConvGeom &g, float *box, int num_sms, cudaStream_t stream);
// the last two in one launch
int layer_sums(const float *wsum, int Cout, const ConvGeom &g, float *sumw_t, float *taps, const float *img, float *box, int num_sms,
               cudaStream_t stream);
int layer_window_sum_adjoint(const float *gsum, const ConvGeom &g, float *out, int num_sms, cudaStream_t stream);
int layer_row_sums(const float *g, long M, int N, float *sums, int num_sms, cudaStream_t stream);
int layer_weight_grad_finish(const float *gwmat, const float *tapg, const float *weight, long s_co, long s_c, long s_h,
                             long s_w, int Cout, int Cin, int kh, int kw, const float *quant, float qmax, float *gw,
                             int num_sms, cudaStream_t stream);

// number of slabs the weight-gradient kernel splits M into (1 = no scratch needed)
int gw_num_splits(int bits, int M, int K, int N, int num_sms);

// with conv.enabled (a convolution whose windows do not overlap) ga is the image gradient gx[B,C,H,W] and every
// (m,k) is written to the position its activation came from; the caller zero-fills gx where nothing lands
int backward_ga(const float *gc, const uint8_t *a, const uint8_t *w, float *ga, const int16_t *lut_ga, int bits,
                int M, int K, int N, const ConvGeom &conv, int num_sms, cudaStream_t stream);

int backward_gw(const float *gc, const uint8_t *a, const uint8_t *w, float *gw, const int16_t *lut_gw, int bits,
                int M, int K, int N, const ConvGeom &conv, float *scratch, int num_splits, int num_sms,
                cudaStream_t stream);

}  // namespace lutgemm
