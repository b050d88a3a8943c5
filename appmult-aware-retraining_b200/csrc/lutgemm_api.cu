// C ABI of liblutgemm_b200.so (declared in include/lutgemm.h): argument validation and dispatch.
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>

#include "lutgemm.h"
#include "lutgemm_common.cuh"
#include "lutgemm_kernels.h"

namespace {

constexpr int kMaxDevices = 64;
int g_num_sms[kMaxDevices];  // 0 = not queried yet; written with the same value by every thread

int current_num_sms() {
    int dev = 0;
    if (!lutgemm::cuda_ok(cudaGetDevice(&dev))) return -1;
    if (dev >= 0 && dev < kMaxDevices && g_num_sms[dev] > 0) return g_num_sms[dev];
    int sms = 0;
    if (!lutgemm::cuda_ok(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) || sms <= 0) return -1;
    if (dev >= 0 && dev < kMaxDevices) g_num_sms[dev] = sms;
    return sms;
}

thread_local char g_msg[256];

// tile fill of a [rows x cols] problem cut into 512 x 64 slab tiles
double slab_fill(long rows, long cols) {
    const long tr = (rows + 511) / 512, tc = (cols + 63) / 64;
    return (double)rows * (double)cols / ((double)tr * 512.0 * (double)tc * 64.0);
}

// tile fill of a [rows x cols] problem cut into 1024 x 32 slab tiles
double tall_fill(long rows, long cols) {
    const long tr = (rows + 1023) / 1024, tc = (cols + 31) / 32;
    return (double)rows * (double)cols / ((double)tr * 1024.0 * (double)tc * 32.0);
}

// kernel-family overrides set through lutgemm_set_kernel_choice (0 = automatic choice by shape)
std::atomic<int> g_force_forward{0}, g_force_backward{0}, g_force_tile{0};

// the CUDA error behind the calling thread's last LUTGEMM_E_CUDA (launchers clear the runtime's own record)
thread_local cudaError_t g_last_cuda_error = cudaSuccess;

// kernels launched by this library in this process (every launch site reports through launch_status)
std::atomic<unsigned long long> g_kernel_launches{0};

struct BackwardPlan {
    bool gw_slab, ga_slab;
    bool gw_tall, ga_tall;  // fp32 slab with the 1024 x 32 tile instead of the packed slab with the 512 x 64 tile
    int gw_splits;        // row-broadcast grad_w kernel: slabs of M
    // slab grad_w kernels read the activation codes from a transposed copy at[k][m] (their row-code fetch is then
    // coalesced; for a convolution it also replaces one implicit-im2col gather per column tile by a single one): the
    // caller's, or one made behind the partial sums in the scratch buffer
    // (grad_a with one thread per row reads them too)
    size_t at_offset;  // bytes into the scratch buffer, a multiple of 16
    int at_pitch;      // 0 = no transposed copy
    size_t scratch;    // whole buffer: sums of either gradient, which run one after the other, then the copy
    lutgemm::PackedPlan gw_packed, ga_packed;
    bool gw_rows, ga_rows;  // one thread per output row instead of the packed or tall slab kernel
    lutgemm::RowsPlan gw_rows_plan, ga_rows_plan;
};

// ---- estimated times of the kernel families, in SM clocks --------------------------------------------------------
// Each estimate is (waves of the kernel's own tiling) x (clocks of one work item) + a fixed start (launch, table staging).
// The clocks are measured on B200, at 4096^3 unless said otherwise:
//   slab kernels, per k and tile      packed 512 x 64: grad_w 1275 (4 bits), 1315 (6), 1365 (7), 1945 (8), grad_a and grad_x
//                                     1290, 1320, 1390, 2055 (grad_x: 9.5e3 more per work item, 2e3 at 8 bits); tall 1024 x 32: 1540, 1690, 1880;
//                                     forward 512 x 64: 905, 940, 1330 and 60e3 / 75e3 at the start (up to three
//                                     more launches: code transposition, zeroing, and a layer's epilogue);
//   a thread per row                  gradients 512 x 64: 1185 (4 bits), 1210 (6 and 7), 1490 (8) per k, 9e3 per block of
//                                     grad_out values (27e3 where they come one by one); forward 1024 x 32: 650, 690, 845
//   broadcast kernels, per 32 look-ups (1 = no bank conflict): forward 1.48, 2.33, 3.1; grad_w 1.6, 2.4, 3.3;
//                                     grad_a 1.6, 2.6, 4.2; grad_x of clustered codes 1.66, 1.7, 2.2
// A slab kernel's time does not depend on the codes and it can cut K into many work items; a broadcast kernel has no slab
// to build, so it stays the better one for few rows.  Against the fixed limits on M, N and tile fill that came before
// (base_plan below) the estimates move small and ragged problems to the slab kernels: 256 x 512 x 256 at 7 bits, forward 0.291 ms,
// grad_w 0.088 ms and grad_a 0.092 ms with the broadcast kernels, both gradients 0.034 ms with the slab kernels.
struct FamilyClocks {
    double packed_gw, packed, tall, fwd_slab, fwd_bcast, gw_bcast, ga_bcast, gx_bcast, fwd_start, rows, fwd_rows;
};
FamilyClocks family_clocks(int bits) {
    if (bits == 8) return {1945, 2055, 1880, 1330, 3.1, 3.3, 4.2, 2.2, 75e3, 1490, 845};
    if (bits == 7) return {1365, 1390, 1690, 940, 2.33, 2.4, 2.6, 1.7, 60e3, 1210, 690};
    if (bits == 6) return {1315, 1320, 1540, 905, 1.48, 1.6, 1.6, 1.66, 60e3, 1210, 650};
    return {1275, 1290, 1540, 905, 1.48, 1.6, 1.6, 1.66, 60e3, 1185, 650};
}
constexpr double kBcastStart = 12e3, kSlabStart = 10e3;
constexpr double kReduceBytesPerClock = 4000;  // reading and writing partial sums, whole GPU

long div_up(long a, long b) { return (a + b - 1) / b; }

double packed_clocks(const lutgemm::PackedPlan &p, long cols, int K, double per_step, bool transposed) {
    const bool reduce = p.groups > 1 || (transposed && p.group_blocks > 1);
    return (double)p.steps * per_step + kSlabStart + (reduce ? 8e3 + 8.0 * p.groups * K * cols / kReduceBytesPerClock : 0);
}
double packed_gw_clocks(const lutgemm::PackedPlan &plan, int bits, int K, int N) {
    return packed_clocks(plan, N, K, family_clocks(bits).packed_gw, false);
}
double packed_ga_clocks(const lutgemm::PackedPlan &plan, int bits, int M, int K, int N) {
    const int rt = lutgemm::packed_ga_tile_rows(N);
    const double step = family_clocks(bits).packed * (rt == 384 ? 0.83 : rt == 576 ? lutgemm::kPacked576Step : 1.0);
    return packed_clocks(plan, M, K, step, true);
}
double tall_clocks(int bits, long rows, long cols, int K, int sms) {
    const long blocks = div_up(rows, 1024);
    const lutgemm::KSplit ks = lutgemm::choose_ksplit(blocks * div_up(cols, 32), K, sms, lutgemm::kTallItemOverhead);
    const double reduce = blocks > 1 ? 8e3 + 8.0 * blocks * K * cols / kReduceBytesPerClock : 0;
    return (double)ks.waves * (ks.per + lutgemm::kTallItemOverhead) * family_clocks(bits).tall + kSlabStart + reduce;
}
double gw_bcast_clocks(int bits, int M, int K, int N, int sms) {
    const long kt = N <= 128 ? 128 : 32, nt = N <= 128 ? 64 : 256, splits = lutgemm::gw_num_splits(bits, M, K, N, sms);
    const long items = div_up(K, kt) * div_up(N, nt) * splits;
    return (double)div_up(items, sms) * kt * nt * div_up(M, splits) * family_clocks(bits).gw_bcast / 32 + kBcastStart +
           (splits > 1 ? 8e3 + 8.0 * splits * K * N / kReduceBytesPerClock : 0);
}
double ga_bcast_clocks(int bits, int M, int K, int N, int sms) {
    const long mt = bits == 8 ? 512 : 256;
    return (double)div_up(div_up(M, mt) * div_up(K, 32), sms) * mt * N * family_clocks(bits).ga_bcast + kBcastStart;
}

// (`aligned`: a block's grad_out values come in 16-byte vectors; `copy`: the transposed codes have to be made for it)
double rows_clocks(const lutgemm::RowsPlan &p, int bits, long rows, int K, bool direct, bool aligned, bool copy) {
    const bool reduce = p.groups > 1 || !direct;
    return p.steps * family_clocks(bits).rows + p.loads * (aligned ? 9e3 : 27e3) + (bits == 8 ? 35e3 : 25e3) + (copy ? 13e3 : 0) +
           (reduce ? 15e3 + 8.0 * p.groups * K * rows / kReduceBytesPerClock : 0);
}

void set_scratch(BackwardPlan &pl, int bits, int M, int K, int N, int sms, bool want_gw, bool want_ga, bool have_codes) {
    size_t gw = 0, ga = 0;
    if (want_gw) {
        pl.gw_splits = pl.gw_slab ? 1 : lutgemm::gw_num_splits(bits, M, K, N, sms);
        const int blocks = !pl.gw_slab ? pl.gw_splits : pl.gw_tall ? lutgemm::slab_tall_row_blocks(M) : pl.gw_packed.groups;
        gw = pl.gw_rows ? lutgemm::rows_scratch_bytes(pl.gw_rows_plan, N, K, true, sms) : blocks > 1 ? (size_t)blocks * K * N * sizeof(float) : 0;
    }
    if (want_ga && pl.ga_slab) {
        const int rt = pl.ga_tall ? lutgemm::kSlabTallRows : lutgemm::packed_ga_tile_rows(N);
        const int blocks = pl.ga_tall ? lutgemm::slab_tall_row_blocks(N) : pl.ga_packed.groups;
        ga = pl.ga_rows ? lutgemm::rows_scratch_bytes(pl.ga_rows_plan, M, K, false, sms) : N > rt ? (size_t)blocks * K * M * sizeof(float) : 0;
    }
    pl.scratch = gw > ga ? gw : ga;
    pl.at_pitch = (want_gw && pl.gw_slab) || (want_ga && pl.ga_rows) ? (M + 15) & ~15 : 0;
    if (pl.at_pitch && !have_codes) {
        pl.at_offset = (pl.scratch + 15) & ~(size_t)15;
        pl.scratch = pl.at_offset + (size_t)pl.at_pitch * K;
    }
}

// Choice by fixed limits: the plan for callers whose scratch buffer is too small for the faster one (a fixed buffer, or
// one sized for this choice), so that what fitted such a buffer keeps running.
BackwardPlan base_plan(int bits, int M, int K, int N, int sms, bool want_gw, bool want_ga, bool have_codes) {
    BackwardPlan pl{};
    pl.gw_slab = bits >= 7 && M >= 512 && N >= 32 && slab_fill(M, N) >= 0.6;
    const double ga_fill = slab_fill(N, M) > tall_fill(N, M) ? slab_fill(N, M) : tall_fill(N, M);
    pl.ga_slab = bits >= 7 && N >= 768 && M >= 32 && ga_fill >= (bits == 7 ? 0.85 : 0.7);
    pl.gw_tall = pl.gw_slab && tall_fill(M, N) >= 0.7 * slab_fill(M, N);
    pl.ga_tall = pl.ga_slab && tall_fill(N, M) >= 0.7 * slab_fill(N, M);
    if (pl.gw_slab && !pl.gw_tall) pl.gw_packed = lutgemm::plan_packed_gw(M, N, K, sms);
    if (pl.ga_slab && !pl.ga_tall) pl.ga_packed = lutgemm::plan_packed(N, M, K, lutgemm::packed_ga_tile_rows(N), sms);
    set_scratch(pl, bits, M, K, N, sms, want_gw, want_ga, have_codes);
    return pl;
}

// Choice by estimated time.  A convolution's grad_a (non-overlapping windows) gathers its column codes from the image and
// writes in place; there the slab kernels pay from N = 768 on (1x1, 128 -> 512 channels, 7 bits: 0.75 against 0.68 ms; 1024 -> 512:
// 1.24 against 1.22 ms).  lutgemm_set_kernel_choice overrides the choice (tests, A/B timing).
// (want_gw, want_ga: the gradients that are asked for; the plan of the other one is left empty.  have_codes: the caller
// brings the transposed activation codes)
BackwardPlan plan_backward(int bits, int M, int K, int N, int sms, bool conv, bool want_gw, bool want_ga, bool have_codes) {
    BackwardPlan pl{};
    const int force = g_force_backward.load(std::memory_order_relaxed), tile = g_force_tile.load(std::memory_order_relaxed);
    const bool rows = tile == LUTGEMM_TILE_ROWS || (!force && !tile);  // may the kernel with one thread per row be chosen?
    if (want_gw) {
        pl.gw_packed = lutgemm::plan_packed_gw(M, N, K, sms);
        const double packed = packed_gw_clocks(pl.gw_packed, bits, K, N), tall = tall_clocks(bits, M, N, K, sms);
        double slab = packed < tall ? packed : tall;
        if (rows && lutgemm::rows_supported(N, M, K)) {
            pl.gw_rows_plan = lutgemm::plan_rows(N, M, K, sms);
            const double t = rows_clocks(pl.gw_rows_plan, bits, N, K, true, N % 4 == 0, false);
            pl.gw_rows = tile == LUTGEMM_TILE_ROWS || t < slab;
            if (pl.gw_rows) slab = t;
        }
        pl.gw_slab = slab < gw_bcast_clocks(bits, M, K, N, sms);
        if (force) pl.gw_slab = force == LUTGEMM_BACKWARD_SLAB;
        pl.gw_rows = pl.gw_rows && pl.gw_slab;
        pl.gw_tall = pl.gw_slab && !pl.gw_rows && (tile ? tile == LUTGEMM_TILE_TALL : tall < packed);
    }
    if (want_ga) {
        pl.ga_packed = lutgemm::plan_packed(N, M, K, lutgemm::packed_ga_tile_rows(N), sms);
        const double packed = packed_ga_clocks(pl.ga_packed, bits, M, K, N), tall = tall_clocks(bits, N, M, K, sms);
        double slab = packed < tall ? packed : tall;
        if (rows && !conv && lutgemm::rows_supported(M, N, K)) {
            pl.ga_rows_plan = lutgemm::plan_rows(M, N, K, sms);
            const double t = rows_clocks(pl.ga_rows_plan, bits, M, K, false, N % 4 == 0, !want_gw && !have_codes);
            pl.ga_rows = tile == LUTGEMM_TILE_ROWS || t < slab;
            if (pl.ga_rows) slab = t;
        }
        pl.ga_slab = (!conv || N >= 768) && slab < ga_bcast_clocks(bits, M, K, N, sms);
        if (force) pl.ga_slab = force == LUTGEMM_BACKWARD_SLAB;
        pl.ga_rows = pl.ga_rows && pl.ga_slab;
        pl.ga_tall = pl.ga_slab && !pl.ga_rows && (tile ? tile == LUTGEMM_TILE_TALL : tall < packed);
    }
    set_scratch(pl, bits, M, K, N, sms, want_gw, want_ga, have_codes);
    return pl;
}

}  // namespace

namespace lutgemm {

void record_cuda_error(cudaError_t e) { g_last_cuda_error = e; }

size_t base_gw_scratch_bytes(int bits, int M, int K, int N) {
    const int sms = current_num_sms();
    if (sms <= 0) return 0;
    if (g_force_backward.load(std::memory_order_relaxed)) return plan_backward(bits, M, K, N, sms, false, true, false, false).scratch;
    return base_plan(bits, M, K, N, sms, true, false, false).scratch;
}

int launch_status() {
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    const cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) return LUTGEMM_OK;
    g_last_cuda_error = e;
    return LUTGEMM_E_CUDA;
}

}  // namespace lutgemm

extern "C" {

int lutgemm_version(void) { return 200; }

const char *lutgemm_status_string(int status) {
    switch (status) {
        case LUTGEMM_OK: return "ok";
        case LUTGEMM_E_BADARG: return "bad argument (null pointer, non-positive size or misaligned buffer)";
        case LUTGEMM_E_BITS: return "unsupported bit-width (supported: 4, 6, 7, 8)";
        case LUTGEMM_E_SCRATCH: return "scratch buffer too small";
        case LUTGEMM_E_TOOLARGE: return "problem size beyond what this entry point supports";
        case LUTGEMM_E_CUDA: {
            snprintf(g_msg, sizeof(g_msg), "CUDA failure: %s", cudaGetErrorString(g_last_cuda_error));
            return g_msg;
        }
    }
    return "unknown status";
}

int lutgemm_set_tma(int on) {
    lutgemm::slab_fwd_set_tma(on != 0);
    return LUTGEMM_OK;
}

int lutgemm_set_handover(int on) {
    lutgemm::slab_tall_set_handover(on != 0);
    return LUTGEMM_OK;
}

unsigned long long lutgemm_kernel_launches(void) { return g_kernel_launches.load(std::memory_order_relaxed); }

int lutgemm_set_kernel_choice(int forward, int backward, int grad_tile) {
    if (forward < 0 || forward > 3 || backward < 0 || backward > 2 || grad_tile < 0 || grad_tile > 3)
        return LUTGEMM_E_BADARG;
    g_force_forward.store(forward, std::memory_order_relaxed);
    g_force_backward.store(backward, std::memory_order_relaxed);
    g_force_tile.store(grad_tile, std::memory_order_relaxed);
    return LUTGEMM_OK;
}

int lutgemm_lut_elem_num(int bits) {
    if (!lutgemm::bits_supported(bits)) return LUTGEMM_E_BITS;
    return lutgemm::lut_elem_num(bits);
}

int lutgemm_bits_from_elem_num(long elem_num) {
    const int all[4] = {4, 6, 7, 8};
    for (int b : all)
        if (lutgemm::lut_elem_num(b) == elem_num) return b;
    return LUTGEMM_E_BITS;
}

// ---- shared bodies of the GEMM and the implicit-im2col entry points ------------------------------------
// The forward kernel by estimated time (see family_clocks); base_forward_uses_slab is the choice by fixed limits, for
// callers whose workspace is too small for it.  lutgemm_set_kernel_choice overrides the choice (tests, A/B timing).
static bool base_forward_uses_slab(int M, int N) { return M >= 512 && N >= 32 && slab_fill(M, N) >= 0.6; }

static double fwd_slab_clocks(int bits, int M, int K, int N, int sms) {
    const FamilyClocks f = family_clocks(bits);
    return (double)div_up(div_up(M, 512) * div_up(N, 64) * div_up(K, 16), sms) * 16 * f.fwd_slab + f.fwd_start;
}
static double fwd_bcast_clocks(int bits, int M, int K, int N, int sms) {
    const long mt = N <= 128 ? 128 : 64, nt = N <= 128 ? 64 : 256;
    return (double)div_up(div_up(M, mt) * div_up(N, nt), sms) * mt * nt * K * family_clocks(bits).fwd_bcast / 32 + kBcastStart;
}
static bool forward_uses_slab(int bits, int M, int K, int N, int sms) {
    const int force = g_force_forward.load(std::memory_order_relaxed);
    if (force == LUTGEMM_FORWARD_ROWBCAST) return false;
    if (force) return true;
    return base_forward_uses_slab(M, N) || fwd_slab_clocks(bits, M, K, N, sms) < fwd_bcast_clocks(bits, M, K, N, sms);
}

// Two rows per thread instead of either, where the caller brings a workspace for the transposed codes: from about a thousand
// rows on (7 bits, slab kernel against two rows per thread, ms: 512^3 0.042 : 0.044, 1000 x 777 x 333 0.067 : 0.052, 1024^3 0.140 :
// 0.108, 200704 x 64 x 256 0.394 : 0.355).
constexpr double kFwdTileClocks = 13e3;  // codes of the first k, sums on their way out
static bool forward_by_rows(int bits, int M, int K, int N, int sms) {
    const int force = g_force_forward.load(std::memory_order_relaxed);
    if (force) return force == LUTGEMM_FORWARD_ROWS;
    const FamilyClocks f = family_clocks(bits);
    const long tiles = div_up(M, lutgemm::kFwdRowsTile) * div_up(N, lutgemm::kFwdRowsCols);
    const bool cut = lutgemm::forward_rows_cut(M, K, N, sms);
    const double k = cut ? 4.0 * div_up(tiles * div_up(K, 4), sms) : (double)div_up(tiles, sms) * K;
    const double t = k * f.fwd_rows + div_up(tiles, sms) * kFwdTileClocks + f.fwd_start;
    return t < fwd_slab_clocks(bits, M, K, N, sms) && (base_forward_uses_slab(M, N) || t < fwd_bcast_clocks(bits, M, K, N, sms));
}

// A workspace too small for the slab kernel is refused where the slab kernel was always the choice (or is forced); elsewhere
// the broadcast kernel, which needs none, runs.
static bool small_workspace_refused(int M, int N) {
    return base_forward_uses_slab(M, N) || g_force_forward.load(std::memory_order_relaxed);
}

static int codes_pitch(int M) { return (M + 15) & ~15; }

// `scratch` (optional, K * codes_pitch(M) bytes, 16-byte aligned): the slab kernels then read the activation
// codes from a transposed copy made there first, which stays valid on return.  `may_rows`: the kernel with two rows per thread
// may be chosen.
static int forward_impl(const uint8_t *a, const uint8_t *w, uint32_t *c, const uint16_t *lut, int bits, int M, int K,
                        int N, const lutgemm::ConvGeom &conv, void *scratch, size_t scratch_bytes, void *stream,
                        const lutgemm::LayerEpilogue *epi = nullptr, bool may_rows = true) {
    if (!lutgemm::bits_supported(bits)) return LUTGEMM_E_BITS;
    if (!a || !w || (!c && !epi) || !lut || M <= 0 || K <= 0 || N <= 0) return LUTGEMM_E_BADARG;
    if ((reinterpret_cast<uintptr_t>(c) & 3) || (reinterpret_cast<uintptr_t>(lut) & 1) ||
        (reinterpret_cast<uintptr_t>(scratch) & 15))
        return LUTGEMM_E_BADARG;
    const int sms = current_num_sms();
    if (sms <= 0) return LUTGEMM_E_CUDA;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int pitch = codes_pitch(M);
    // the copy's launch sets the sums to zero where its M * K / 16 threads have 64 words each at most
    const bool few_sums = N <= 4 * (long)K;
    if (may_rows && scratch && scratch_bytes >= (size_t)pitch * K && forward_by_rows(bits, M, K, N, sms)) {
        const bool zero = few_sums && !epi && lutgemm::forward_rows_cut(M, K, N, sms);
        const int trc = lutgemm::transpose_codes(a, static_cast<uint8_t *>(scratch), M, K, pitch, conv, bits, zero ? c : nullptr, (long)M * N, s);
        if (trc != LUTGEMM_OK) return trc;
        return lutgemm::forward_rows(w, c, lut, bits, M, K, N, static_cast<const uint8_t *>(scratch), pitch, epi, zero, sms, s);
    }
    bool slab = forward_uses_slab(bits, M, K, N, sms);
    if (slab && scratch && scratch_bytes < (size_t)pitch * K) {
        if (small_workspace_refused(M, N)) return LUTGEMM_E_SCRATCH;
        slab = false;
    }
    if (slab) {
        const uint8_t *at = nullptr;
        const bool zero = scratch && few_sums && !epi && lutgemm::slab_fwd_ksplits(M, K, N, sms) > 1;
        if (scratch) {
            const int trc = lutgemm::transpose_codes(a, static_cast<uint8_t *>(scratch), M, K, pitch, conv, bits, zero ? c : nullptr, (long)M * N, s);
            if (trc != LUTGEMM_OK) return trc;
            at = static_cast<const uint8_t *>(scratch);
        }
        return lutgemm::forward_slab(a, w, c, lut, bits, M, K, N, conv, at, pitch, epi, zero, sms, s);
    }
    return lutgemm::forward_rowbcast(a, w, c, lut, bits, M, K, N, conv, epi, sms, s);
}

int lutgemm_forward(const uint8_t *a, const uint8_t *w, uint32_t *c, const uint16_t *lut, int bits, int M, int K,
                    int N, void *stream) {
    lutgemm::ConvGeom none{};
    return forward_impl(a, w, c, lut, bits, M, K, N, none, nullptr, 0, stream);
}

size_t lutgemm_forward_scratch_bytes(int bits, int M, int K, int N) {
    if (!lutgemm::bits_supported(bits) || M <= 0 || K <= 0 || N <= 0) return 0;
    const int sms = current_num_sms();
    if (sms <= 0 || !(forward_uses_slab(bits, M, K, N, sms) || forward_by_rows(bits, M, K, N, sms))) return 0;
    return (size_t)codes_pitch(M) * K;
}

int lutgemm_forward_ws(const uint8_t *a, const uint8_t *w, uint32_t *c, const uint16_t *lut, int bits, int M, int K,
                       int N, void *scratch, size_t scratch_bytes, void *stream) {
    lutgemm::ConvGeom none{};
    return forward_impl(a, w, c, lut, bits, M, K, N, none, scratch, scratch_bytes, stream);
}

int lutgemm_device_error(int *value) {
    if (!value) return LUTGEMM_E_BADARG;
    return lutgemm::read_and_clear_device_error(value);
}

int lutgemm_selftest_bounded_wait(void *stream) {
    return lutgemm::bounded_wait_selftest(static_cast<cudaStream_t>(stream));
}

// of a buffer for the faster choice and one for the fixed limits, the smaller one that is accepted
static size_t least_need(size_t need, size_t base) {
    return base < need && !g_force_backward.load(std::memory_order_relaxed) ? base : need;
}

size_t lutgemm_backward_ws_scratch_bytes(int bits, int M, int K, int N, int flags) {
    if (!lutgemm::bits_supported(bits) || M <= 0 || K <= 0 || N <= 0) return 0;
    const int sms = current_num_sms();
    if (sms <= 0) return 0;
    const bool have_codes = flags & LUTGEMM_SCRATCH_CODES_GIVEN;
    const BackwardPlan both = plan_backward(bits, M, K, N, sms, false, true, true, have_codes);
    size_t need = both.scratch;
    if (both.ga_rows && !have_codes) {  // (alone, grad_a has the code copy made for itself and may choose another kernel)
        const size_t alone = plan_backward(bits, M, K, N, sms, false, false, true, false).scratch;
        need = alone > need ? alone : need;
    }
    return flags & LUTGEMM_SCRATCH_LEAST ? least_need(need, base_plan(bits, M, K, N, sms, true, true, have_codes).scratch) : need;
}

size_t lutgemm_backward_scratch_bytes(int bits, int M, int K, int N) {
    return lutgemm_backward_ws_scratch_bytes(bits, M, K, N, 0);
}

static int backward_impl(const float *gc, const uint8_t *a, const uint8_t *w, float *ga, float *gw,
                         const int16_t *lut_ga, const int16_t *lut_gw, int bits, int M, int K, int N,
                         const lutgemm::ConvGeom &conv, const uint8_t *codes_t, void *scratch, size_t scratch_bytes,
                         void *stream) {
    if (!lutgemm::bits_supported(bits)) return LUTGEMM_E_BITS;
    if (!gc || !a || !w || M <= 0 || K <= 0 || N <= 0) return LUTGEMM_E_BADARG;
    if ((ga && !lut_ga) || (gw && !lut_gw)) return LUTGEMM_E_BADARG;
    if ((reinterpret_cast<uintptr_t>(gc) & 3) || (reinterpret_cast<uintptr_t>(ga) & 3) ||
        (reinterpret_cast<uintptr_t>(gw) & 3) || (reinterpret_cast<uintptr_t>(scratch) & 15) ||
        (reinterpret_cast<uintptr_t>(lut_ga) & 1) || (reinterpret_cast<uintptr_t>(lut_gw) & 1))
        return LUTGEMM_E_BADARG;
    const int sms = current_num_sms();
    if (sms <= 0) return LUTGEMM_E_CUDA;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const size_t given = scratch ? scratch_bytes : 0;
    BackwardPlan pl = plan_backward(bits, M, K, N, sms, conv.enabled != 0, gw != nullptr, ga != nullptr, codes_t != nullptr);
    if (pl.scratch > given && !g_force_backward.load(std::memory_order_relaxed))
        pl = base_plan(bits, M, K, N, sms, gw != nullptr, ga != nullptr, codes_t != nullptr);
    if (pl.scratch > given) return LUTGEMM_E_SCRATCH;
    float *sc = static_cast<float *>(scratch);
    const uint8_t *at = codes_t;  // left by the forward pass (same layout), or made here
    if (pl.at_pitch && !at) {
        uint8_t *dst = static_cast<uint8_t *>(scratch) + pl.at_offset;
        const int trc = lutgemm::transpose_codes(a, dst, M, K, pl.at_pitch, conv, bits, nullptr, 0, s);
        if (trc != LUTGEMM_OK) return trc;
        at = dst;
    }
    if (gw) {
        // the weight gradient goes first: under data parallelism its all-reduce can then overlap gA
        int rc = !pl.gw_slab ? lutgemm::backward_gw(gc, a, w, gw, lut_gw, bits, M, K, N, conv, sc, pl.gw_splits, sms, s)
                 : pl.gw_rows ? lutgemm::backward_gw_rows(gc, w, gw, lut_gw, bits, M, K, N, pl.gw_rows_plan, sc, at, pl.at_pitch, sms, s)
                 : pl.gw_tall ? lutgemm::backward_gw_slab_tall(gc, a, w, gw, lut_gw, nullptr, bits, M, K, N, conv, sc, at, pl.at_pitch, sms, s)
                             : lutgemm::backward_gw_slab_packed(gc, a, w, gw, lut_gw, bits, M, K, N, conv, pl.gw_packed, sc, at, pl.at_pitch, sms, s);
        if (rc != LUTGEMM_OK) return rc;
    }
    if (ga) {
        int rc = !pl.ga_slab ? lutgemm::backward_ga(gc, a, w, ga, lut_ga, bits, M, K, N, conv, sms, s)
                 : pl.ga_rows ? lutgemm::backward_ga_rows(gc, w, ga, lut_ga, bits, M, K, N, pl.ga_rows_plan, sc, at, pl.at_pitch, sms, s)
                 : pl.ga_tall ? lutgemm::backward_ga_slab_tall(gc, a, w, ga, lut_ga, nullptr, bits, M, K, N, conv, sc, sms, s)
                             : lutgemm::backward_ga_slab_packed(gc, a, w, ga, lut_ga, bits, M, K, N, conv, pl.ga_packed, sc, sms, s);
        if (rc != LUTGEMM_OK) return rc;
    }
    return LUTGEMM_OK;
}

int lutgemm_backward(const float *gc, const uint8_t *a, const uint8_t *w, float *ga, float *gw,
                     const int16_t *lut_ga, const int16_t *lut_gw, int bits, int M, int K, int N, void *scratch,
                     size_t scratch_bytes, void *stream) {
    lutgemm::ConvGeom none{};
    return backward_impl(gc, a, w, ga, gw, lut_ga, lut_gw, bits, M, K, N, none, nullptr, scratch, scratch_bytes, stream);
}

int lutgemm_backward_ws(const float *gc, const uint8_t *a, const uint8_t *w, float *ga, float *gw,
                        const int16_t *lut_ga, const int16_t *lut_gw, int bits, int M, int K, int N,
                        const uint8_t *codes_t, void *scratch, size_t scratch_bytes, void *stream) {
    if (reinterpret_cast<uintptr_t>(codes_t) & 15) return LUTGEMM_E_BADARG;
    lutgemm::ConvGeom none{};
    return backward_impl(gc, a, w, ga, gw, lut_ga, lut_gw, bits, M, K, N, none, codes_t, scratch, scratch_bytes, stream);
}

// ---- gradient tables in fp32 (bits <= 7) -------------------------------------------------------------------------
// Always the tall slab kernels: their fp32 shared-memory table takes either entry type; tiles of small problems
// are mostly empty, which costs time, not correctness.
size_t lutgemm_backward_f32lut_scratch_bytes(int bits, int M, int K, int N) {
    if (!lutgemm::bits_supported(bits) || bits > 7 || M <= 0 || K <= 0 || N <= 0) return 0;
    const size_t rb_w = lutgemm::slab_tall_row_blocks(M), rb_a = lutgemm::slab_tall_row_blocks(N);
    const size_t gw_need = rb_w > 1 ? rb_w * K * N * sizeof(float) : 0;
    const size_t ga_need = rb_a > 1 ? rb_a * K * M * sizeof(float) : 0;
    return gw_need > ga_need ? gw_need : ga_need;
}

int lutgemm_backward_f32lut(const float *gc, const uint8_t *a, const uint8_t *w, float *ga, float *gw,
                            const float *lut_ga, const float *lut_gw, int bits, int M, int K, int N, void *scratch,
                            size_t scratch_bytes, void *stream) {
    if (!lutgemm::bits_supported(bits) || bits > 7) return LUTGEMM_E_BITS;
    if (!gc || !a || !w || M <= 0 || K <= 0 || N <= 0) return LUTGEMM_E_BADARG;
    if ((ga && !lut_ga) || (gw && !lut_gw)) return LUTGEMM_E_BADARG;
    if ((reinterpret_cast<uintptr_t>(gc) & 3) || (reinterpret_cast<uintptr_t>(ga) & 3) ||
        (reinterpret_cast<uintptr_t>(gw) & 3) || (reinterpret_cast<uintptr_t>(scratch) & 15) ||
        (reinterpret_cast<uintptr_t>(lut_ga) & 3) || (reinterpret_cast<uintptr_t>(lut_gw) & 3))
        return LUTGEMM_E_BADARG;
    if (lutgemm_backward_f32lut_scratch_bytes(bits, M, K, N) > (scratch ? scratch_bytes : 0)) return LUTGEMM_E_SCRATCH;
    const int sms = current_num_sms();
    if (sms <= 0) return LUTGEMM_E_CUDA;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    lutgemm::ConvGeom none{};
    float *sc = static_cast<float *>(scratch);
    if (gw) {
        const int rc = lutgemm::backward_gw_slab_tall(gc, a, w, gw, nullptr, lut_gw, bits, M, K, N, none, sc, nullptr, 0, sms, s);
        if (rc != LUTGEMM_OK) return rc;
    }
    if (ga) {
        const int rc = lutgemm::backward_ga_slab_tall(gc, a, w, ga, nullptr, lut_ga, bits, M, K, N, none, sc, sms, s);
        if (rc != LUTGEMM_OK) return rc;
    }
    return LUTGEMM_OK;
}

// ---- convolution entry points (implicit im2col) ------------------------------------------------------------
static int make_geom(int B, int C, int H, int W, int kh, int kw, int stride, int pad, int dil, lutgemm::ConvGeom *g) {
    if (B <= 0 || C <= 0 || H <= 0 || W <= 0 || kh <= 0 || kw <= 0 || stride <= 0 || pad < 0 || dil <= 0)
        return LUTGEMM_E_BADARG;
    const long Ho = ((long)H + 2L * pad - (long)dil * (kh - 1) - 1) / stride + 1;
    const long Wo = ((long)W + 2L * pad - (long)dil * (kw - 1) - 1) / stride + 1;
    if (Ho <= 0 || Wo <= 0) return LUTGEMM_E_BADARG;
    if ((long)B * Ho * Wo > 0x7fffffffL || (long)C * kh * kw > 0x7fffffffL) return LUTGEMM_E_TOOLARGE;
    g->enabled = 1; g->B = B; g->C = C; g->H = H; g->W = W; g->kh = kh; g->kw = kw;
    g->stride = stride; g->pad = pad; g->dil = dil; g->Ho = (int)Ho; g->Wo = (int)Wo;
    return LUTGEMM_OK;
}

int lutgemm_conv2d_forward(const uint8_t *x, const uint8_t *wmat, uint32_t *y, const uint16_t *lut, int bits, int B,
                           int C, int H, int W, int Cout, int kh, int kw, int stride, int pad, int dil,
                           void *stream) {
    lutgemm::ConvGeom g{};
    const int rc = make_geom(B, C, H, W, kh, kw, stride, pad, dil, &g);
    if (rc != LUTGEMM_OK) return rc;
    return forward_impl(x, wmat, y, lut, bits, B * g.Ho * g.Wo, C * kh * kw, Cout, g, nullptr, 0, stream);
}

size_t lutgemm_conv2d_forward_scratch_bytes(int bits, int B, int C, int H, int W, int Cout, int kh, int kw,
                                            int stride, int pad, int dil) {
    lutgemm::ConvGeom g{};
    if (make_geom(B, C, H, W, kh, kw, stride, pad, dil, &g) != LUTGEMM_OK) return 0;
    return lutgemm_forward_scratch_bytes(bits, B * g.Ho * g.Wo, C * kh * kw, Cout);
}

int lutgemm_conv2d_forward_ws(const uint8_t *x, const uint8_t *wmat, uint32_t *y, const uint16_t *lut, int bits, int B,
                              int C, int H, int W, int Cout, int kh, int kw, int stride, int pad, int dil,
                              void *scratch, size_t scratch_bytes, void *stream) {
    lutgemm::ConvGeom g{};
    const int rc = make_geom(B, C, H, W, kh, kw, stride, pad, dil, &g);
    if (rc != LUTGEMM_OK) return rc;
    return forward_impl(x, wmat, y, lut, bits, B * g.Ho * g.Wo, C * kh * kw, Cout, g, scratch, scratch_bytes, stream);
}

// ---- activation gradient of a convolution ------------------------------------------------------------------
// Windows that do not overlap (kernel extent <= stride, e.g. 1x1 convolutions and patch embeddings): every image
// position receives at most one (m,k) term, so the GEMM-shaped grad_a kernels write it in place.  Overlapping
// windows: the pixel-mode slab kernel, one launch per stride class (lutgemm_slab_grad.cu).  Either way no
// unfolded gradient [M,K] exists.
static bool conv_windows_overlap(const lutgemm::ConvGeom &g) {
    return g.dil * (g.kh - 1) + 1 > g.stride || g.dil * (g.kw - 1) + 1 > g.stride;
}

// the stride class (ph, pw) of geometry g; false when the class has no pixels, no taps or more than it can hold
static bool make_pixel_class(const lutgemm::ConvGeom &g, int ph, int pw, lutgemm::PixelClass *px) {
    *px = lutgemm::PixelClass{};
    px->H = g.H; px->W = g.W; px->C = g.C; px->ph = ph; px->pw = pw; px->s = g.stride; px->Ho = g.Ho; px->Wo = g.Wo;
    px->T = g.kh * g.kw;
    px->Hc = ph < g.H ? (g.H - ph + g.stride - 1) / g.stride : 0;
    px->Wc = pw < g.W ? (g.W - pw + g.stride - 1) / g.stride : 0;
    int n = 0;
    for (int i = 0; i < g.kh; ++i)
        for (int j = 0; j < g.kw; ++j) {
            const int dh = i * g.dil - g.pad, dw = j * g.dil - g.pad;
            const int rh = (((ph - dh) % g.stride) + g.stride) % g.stride, rw = (((pw - dw) % g.stride) + g.stride) % g.stride;
            if (rh != 0 || rw != 0) continue;
            if (n == lutgemm::kMaxTaps) return false;
            px->dh[n] = (int8_t)dh; px->dw[n] = (int8_t)dw; px->t[n] = (uint8_t)(i * g.kw + j);
            ++n;
        }
    px->ntaps = n;
    px->P = g.B * px->Hc * px->Wc;
    return n > 0 && px->Hc > 0 && px->Wc > 0;
}

// pixel mode is limited by the tap tables of PixelClass
static bool pixel_mode_supported(const lutgemm::ConvGeom &g) {
    const int max_d = (g.kh > g.kw ? g.kh : g.kw) * g.dil;
    return g.kh * g.kw <= lutgemm::kMaxTaps && g.kh * g.kw <= 256 && max_d <= 127 && g.pad <= 127;
}

// f(class) for every stride class of the convolution that has pixels and taps
extern "C++" {
template <typename F>
static void for_each_pixel_class(const lutgemm::ConvGeom &g, F f) {
    lutgemm::PixelClass px;
    for (int ph = 0; ph < g.stride; ++ph)
        for (int pw = 0; pw < g.stride; ++pw)
            if (make_pixel_class(g, ph, pw, &px)) f(px);
}
}

// Slab kernel in pixel mode (rows = taps * Cout) or column-broadcast gather kernel in pixel mode, by estimated time (see
// family_clocks).  The slab kernel's time does not depend on the codes, the broadcast kernel's bank conflicts do; the
// estimate takes the clustered codes of a trained layer.  Measured on B200, 3x3 layers at batch 256, clustered codes,
// broadcast against slab, ms:
//   7 bits  64 channels (576 rows) 1.79 : 1.79   128 (1152) 1.99 : 1.60   256 (2304) 2.00 : 1.55   512 (4608) 2.00 : 1.49
//   8 bits  64 channels            2.27 : 2.49   128        2.55 : 2.32   256        2.55 : 2.23   512        2.57 : 2.26
//   stride 2, 128 -> 256 channels: 7 bits 1.03 : 0.99, 8 bits 1.31 : 1.42; 256 -> 512 (classes of 2048, 1024, 1024 and 512 rows):
//   7 bits 1.08 : 0.88, 8 bits 1.73 : 1.30
// or, for callers that allow it (`rows`), the kernel with one thread per pixel (lutgemm_slab_rows.cu).
// (the kernel with a thread per pixel addresses an image by 32-bit offsets and keeps the two coordinates of a pixel in one word)
static bool gx_rows_supported(const lutgemm::ConvGeom &g, int Cout) {
    return g.H < 32768 && g.W < 65536 && (double)g.B * g.C * g.H * g.W < 4294967296.0 && lutgemm::rows_supported((long)g.B * g.H * g.W, (long)g.kh * g.kw * Cout, g.C);
}
struct GxTimes {
    double slab, bcast, rows;  // rows: 0 where that kernel is no choice
    size_t slab_bytes, rows_bytes;
};
static GxTimes gx_times(int bits, const lutgemm::ConvGeom &g, int Cout, int sms, bool rows_allowed) {
    const FamilyClocks f = family_clocks(bits);
    const long mt = bits == 8 ? 512 : 256;
    const bool may_rows = rows_allowed && gx_rows_supported(g, Cout);
    GxTimes times{};
    // broadcast kernel: tiles of all classes in one list, tile t on SM t mod sms (rows_of[i] rows from tile begin[i] on)
    constexpr int kMaxListed = 16;
    long begin[kMaxListed + 1] = {0}, rows_of[kMaxListed], most = 0;
    int n = 0;
    for_each_pixel_class(g, [&](const lutgemm::PixelClass &px) {
        const long rows = (long)px.ntaps * Cout, t = div_up(px.P, mt) * div_up(px.C, 32);
        const int rt = lutgemm::gx_tile_rows(rows);
        const lutgemm::PackedPlan plan = lutgemm::plan_packed(rows, px.P, px.C, rt, sms);
        times.slab += packed_clocks(plan, px.P, px.C, f.packed * (rt > 512 ? lutgemm::kPacked576Step : 1.0), false) + plan.items * (bits == 8 ? 2e3 : 9.5e3);
        times.slab_bytes = std::max(times.slab_bytes, lutgemm::gx_class_scratch_bytes(plan, px));
        if (may_rows) {
            const lutgemm::RowsPlan by_rows = lutgemm::plan_rows(px.P, rows, px.C, sms);
            times.rows += rows_clocks(by_rows, bits, px.P, px.C, true, Cout % 4 == 0, false);
            times.rows_bytes = std::max(times.rows_bytes, lutgemm::rows_scratch_bytes(by_rows, px.P, px.C, true, sms));
        }
        if (n == kMaxListed) {  // (more stride classes than this: the rest counts as tiles of the last one)
            begin[n] += t;
            return;
        }
        rows_of[n] = rows;
        begin[n + 1] = begin[n] + t;
        ++n;
    });
    // what an SM gets changes only at the SMs where a class begins or ends, SM 0 (class 0) among them
    for (int i = 0; i < n; ++i) {
        const long sm = begin[i] % sms;
        long rows = 0;
        for (int c = 0; c < n; ++c) rows += rows_of[c] * ((begin[c + 1] + sms - 1 - sm) / sms - (begin[c] + sms - 1 - sm) / sms);
        if (rows > most) most = rows;
    }
    times.bcast = (double)most * mt * f.gx_bcast + kBcastStart;
    return times;
}
enum GxFamily { kGxBcast, kGxSlab, kGxRows };
static GxFamily gx_family(const GxTimes &t, bool rows) {
    rows = rows && t.rows > 0;
    const int force = g_force_backward.load(std::memory_order_relaxed), tile = g_force_tile.load(std::memory_order_relaxed);
    if (force == LUTGEMM_BACKWARD_BCAST) return kGxBcast;
    if (force == LUTGEMM_BACKWARD_SLAB) return rows && tile == LUTGEMM_TILE_ROWS ? kGxRows : kGxSlab;
    if (rows && t.rows < t.slab && t.rows < t.bcast) return kGxRows;
    return t.slab < t.bcast ? kGxSlab : kGxBcast;
}

// Scratch that the choice by fixed limits (see base_plan) asked for: a buffer of at least that size is not refused, the
// broadcast kernel, which needs none, runs where the slab kernel's partial sums do not fit.
static size_t gx_base_scratch_bytes(int bits, const lutgemm::ConvGeom &g, int Cout) {
    size_t need = 0;
    for_each_pixel_class(g, [&](const lutgemm::PixelClass &px) {
        const long rows = (long)px.ntaps * Cout;
        if (!(bits == 7 ? rows >= 8192 : bits == 8 && (rows >= 4096 || Cout >= 512))) return;
        auto cost = [&](long rt) { return div_up(rows, rt) * (rt + (bits == 8 ? 384 : 256)); };
        long rt = 1024;
        for (long cand : {576L, 512L})
            if (cost(cand) < cost(rt)) rt = cand;
        const long blocks = div_up(rows, rt);
        const size_t n = blocks > 1 ? (size_t)blocks * px.C * px.P * sizeof(float) : 0;
        need = n > need ? n : need;
    });
    return need;
}

// 1x1 windows without padding: every pixel of class (0, 0), of which there are as many as output positions, has the one tap
static bool pointwise(const lutgemm::ConvGeom &g) { return g.kh == 1 && g.kw == 1 && g.pad == 0; }
static bool pointwise_by_rows(int bits, const lutgemm::ConvGeom &g, int Cout, int sms, size_t *bytes) {
    const int force = g_force_backward.load(std::memory_order_relaxed), tile = g_force_tile.load(std::memory_order_relaxed);
    if (!pointwise(g) || force == LUTGEMM_BACKWARD_BCAST || !gx_rows_supported(g, Cout)) return false;
    const int M = g.B * g.Ho * g.Wo;
    const lutgemm::RowsPlan plan = lutgemm::plan_rows(M, Cout, g.C, sms);
    *bytes = lutgemm::rows_scratch_bytes(plan, M, g.C, true, sms);
    if (force || tile) return tile == LUTGEMM_TILE_ROWS;
    const double rows = rows_clocks(plan, bits, M, g.C, true, Cout % 4 == 0, false);
    double best = ga_bcast_clocks(bits, M, g.C, Cout, sms);
    if (Cout >= 768) {
        const lutgemm::PackedPlan pp = lutgemm::plan_packed(Cout, M, g.C, lutgemm::packed_ga_tile_rows(Cout), sms);
        const double packed = packed_ga_clocks(pp, bits, M, g.C, Cout), tall = tall_clocks(bits, Cout, M, g.C, sms);
        best = packed < best ? packed : best;
        best = tall < best ? tall : best;
    }
    return rows < best;
}

static size_t conv_gx_scratch_bytes(int bits, const lutgemm::ConvGeom &g, int Cout) {
    const int M = g.B * g.Ho * g.Wo, K = g.C * g.kh * g.kw;
    const int sms = current_num_sms();
    if (sms <= 0) return 0;
    if (conv_windows_overlap(g) && !pixel_mode_supported(g)) return 0;  // the gradient is refused, whatever the buffer
    // (either entry point's choice, see lutgemm_conv2d_backward)
    if (!conv_windows_overlap(g)) {
        const size_t need = plan_backward(bits, M, K, Cout, sms, true, false, true, false).scratch;
        size_t rows = 0;
        return pointwise_by_rows(bits, g, Cout, sms, &rows) ? std::max(need, rows) : need;
    }
    const GxTimes t = gx_times(bits, g, Cout, sms, true);
    return std::max(gx_family(t, false) == kGxSlab ? t.slab_bytes : 0, gx_family(t, true) == kGxRows ? t.rows_bytes : 0);
}

size_t lutgemm_conv2d_backward_ws_scratch_bytes(int bits, int B, int C, int H, int W, int Cout, int kh, int kw,
                                                int stride, int pad, int dil, int flags) {
    lutgemm::ConvGeom g{};
    if (!lutgemm::bits_supported(bits) || Cout <= 0 || make_geom(B, C, H, W, kh, kw, stride, pad, dil, &g) != LUTGEMM_OK)
        return 0;
    const int sms = current_num_sms();
    if (sms <= 0) return 0;
    const int M = B * g.Ho * g.Wo, K = C * kh * kw;
    // the weight-gradient and the activation-gradient kernels run one after the other on the same buffer
    const bool have_codes = flags & LUTGEMM_SCRATCH_CODES_GIVEN;
    size_t gw_need = plan_backward(bits, M, K, Cout, sms, true, true, false, have_codes).scratch;
    size_t gx_need = conv_gx_scratch_bytes(bits, g, Cout);
    if (flags & LUTGEMM_SCRATCH_LEAST) {
        gw_need = least_need(gw_need, base_plan(bits, M, K, Cout, sms, true, false, have_codes).scratch);
        gx_need = least_need(gx_need, conv_windows_overlap(g) ? gx_base_scratch_bytes(bits, g, Cout)
                                                              : base_plan(bits, M, K, Cout, sms, false, true, have_codes).scratch);
    }
    return gw_need > gx_need ? gw_need : gx_need;
}

size_t lutgemm_conv2d_backward_scratch_bytes(int bits, int B, int C, int H, int W, int Cout, int kh, int kw,
                                             int stride, int pad, int dil) {
    return lutgemm_conv2d_backward_ws_scratch_bytes(bits, B, C, H, W, Cout, kh, kw, stride, pad, dil, 0);
}

// `by_rows`: the image gradient may be computed with one thread per pixel
static int conv_backward_impl(const float *gy, const uint8_t *x, const uint8_t *wmat, float *gx, float *gw,
                              const int16_t *lut_ga, const int16_t *lut_gw, int bits, int B, int C, int H, int W,
                              int Cout, int kh, int kw, int stride, int pad, int dil, const uint8_t *codes_t,
                              void *scratch, size_t scratch_bytes, void *stream, bool by_rows) {
    lutgemm::ConvGeom g{};
    int rc = make_geom(B, C, H, W, kh, kw, stride, pad, dil, &g);
    if (rc != LUTGEMM_OK) return rc;
    if (reinterpret_cast<uintptr_t>(codes_t) & 15) return LUTGEMM_E_BADARG;
    if (gx && !lut_ga) return LUTGEMM_E_BADARG;
    const int M = B * g.Ho * g.Wo, K = C * kh * kw;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (gw) {
        // first, so that under data parallelism its all-reduce can overlap the activation gradient
        rc = backward_impl(gy, x, wmat, nullptr, gw, nullptr, lut_gw, bits, M, K, Cout, g, codes_t, scratch, scratch_bytes,
                           stream);
        if (rc != LUTGEMM_OK) return rc;
    }
    if (!gx) return LUTGEMM_OK;
    if (!lutgemm::bits_supported(bits)) return LUTGEMM_E_BITS;
    if (!gy || !x || !wmat || Cout <= 0) return LUTGEMM_E_BADARG;
    if ((reinterpret_cast<uintptr_t>(gx) & 3) || (reinterpret_cast<uintptr_t>(scratch) & 15)) return LUTGEMM_E_BADARG;
    const bool overlap = conv_windows_overlap(g);
    const bool every_pixel_written = overlap ? stride == 1 : (stride == 1 && kh == 1 && kw == 1 && pad == 0);
    if (!every_pixel_written &&
        !lutgemm::cuda_ok(cudaMemsetAsync(gx, 0, (size_t)B * C * H * W * sizeof(float), s)))
        return LUTGEMM_E_CUDA;
    const int sms = current_num_sms();
    if (sms <= 0) return LUTGEMM_E_CUDA;
    const size_t given = scratch ? scratch_bytes : 0;
    GxFamily family = kGxBcast;
    if (!overlap) {  // conv.enabled makes the grad_a kernels write (m,k) to the image position it came from
        size_t need = 0;
        if (!by_rows || !pointwise_by_rows(bits, g, Cout, sms, &need) || need > given)
            return backward_impl(gy, x, wmat, gx, nullptr, lut_ga, nullptr, bits, M, K, Cout, g, nullptr, scratch, scratch_bytes,
                                 stream);
        family = kGxRows;
    } else {
        if (!pixel_mode_supported(g)) return LUTGEMM_E_TOOLARGE;
        const GxTimes t = gx_times(bits, g, Cout, sms, by_rows);
        family = gx_family(t, by_rows);
        if (family == kGxRows && t.rows_bytes > given) family = gx_family(t, false);
        if (family == kGxSlab && t.slab_bytes > given) {
            if (g_force_backward.load(std::memory_order_relaxed) || gx_base_scratch_bytes(bits, g, Cout) > given)
                return LUTGEMM_E_SCRATCH;
            family = kGxBcast;
        }
    }
    lutgemm::PixelClass px;
    lutgemm::PixelClass bcast[lutgemm::kMaxClassesPerLaunch];  // classes for the broadcast kernel, launched in groups
    int nb = 0;
    for (int ph = 0; ph < stride; ++ph)
        for (int pw = 0; pw < stride; ++pw) {
            if (!make_pixel_class(g, ph, pw, &px)) continue;
            if (family == kGxRows) {
                rc = lutgemm::backward_gx_rows(gy, x, wmat, gx, lut_ga, bits, Cout, px, static_cast<float *>(scratch), sms, s);
                if (rc != LUTGEMM_OK) return rc;
                continue;
            }
            if (family == kGxSlab) {
                rc = lutgemm::backward_gx_class(gy, x, wmat, gx, lut_ga, bits, Cout, px, B, static_cast<float *>(scratch), sms, s);
                if (rc != LUTGEMM_OK) return rc;
                continue;
            }
            bcast[nb++] = px;
            if (nb == lutgemm::kMaxClassesPerLaunch) {
                rc = lutgemm::backward_gx_bcast(gy, x, wmat, gx, lut_ga, bits, Cout, bcast, nb, sms, s);
                if (rc != LUTGEMM_OK) return rc;
                nb = 0;
            }
        }
    if (nb) return lutgemm::backward_gx_bcast(gy, x, wmat, gx, lut_ga, bits, Cout, bcast, nb, sms, s);
    return LUTGEMM_OK;
}

int lutgemm_conv2d_backward_ws(const float *gy, const uint8_t *x, const uint8_t *wmat, float *gx, float *gw,
                               const int16_t *lut_ga, const int16_t *lut_gw, int bits, int B, int C, int H, int W,
                               int Cout, int kh, int kw, int stride, int pad, int dil, const uint8_t *codes_t,
                               void *scratch, size_t scratch_bytes, void *stream) {
    return conv_backward_impl(gy, x, wmat, gx, gw, lut_ga, lut_gw, bits, B, C, H, W, Cout, kh, kw, stride, pad, dil, codes_t,
                              scratch, scratch_bytes, stream, true);
}

// (the tests hold its image gradients to the packed and the broadcast kernel; by the same estimates, so that the one query serves
// both entry points)
int lutgemm_conv2d_backward(const float *gy, const uint8_t *x, const uint8_t *wmat, float *gx, float *gw,
                            const int16_t *lut_ga, const int16_t *lut_gw, int bits, int B, int C, int H, int W,
                            int Cout, int kh, int kw, int stride, int pad, int dil, void *scratch,
                            size_t scratch_bytes, void *stream) {
    return conv_backward_impl(gy, x, wmat, gx, gw, lut_ga, lut_gw, bits, B, C, H, W, Cout, kh, kw, stride, pad, dil, nullptr,
                              scratch, scratch_bytes, stream, false);
}

// ---- forward with the layer's de-quantisation applied where the kernel stores ------------------------------------
static int make_epilogue(const float *box, const float *sumw_t, const float *taps, const float *s_a, const float *s_w,
                         const float *z_a, const float *z_w, const float *bias, float *out, int L,
                         lutgemm::LayerEpilogue *e) {
    if (!box || !sumw_t || !taps || !s_a || !s_w || !z_a || !z_w || !out || L <= 0) return LUTGEMM_E_BADARG;
    if (reinterpret_cast<uintptr_t>(out) & 3) return LUTGEMM_E_BADARG;
    e->box = box; e->sumw_t = sumw_t; e->taps = taps; e->s_a = s_a; e->s_w = s_w; e->z_a = z_a; e->z_w = z_w;
    e->bias = bias; e->out = out; e->L = L;
    return LUTGEMM_OK;
}

// Shared body: with complete sums per tile the de-quantisation runs where the kernel stores; when cutting K across
// CTAs fills the GPU better (few output tiles), the sums go through a uint32 buffer behind the transposed codes in
// `scratch` and the one-pass epilogue kernel finishes them.
static size_t align16(size_t n) { return (n + 15) & ~(size_t)15; }

static bool layer_forward_needs_sums(int bits, int M, int K, int N, int sms) {
    return forward_uses_slab(bits, M, K, N, sms) && lutgemm::slab_fwd_ksplits(M, K, N, sms) > 1;
}

// what the layer forward pass needs at least where it refuses a smaller buffer
static size_t layer_forward_base_bytes(int bits, int M, int K, int N, int sms) {
    const size_t codes = forward_uses_slab(bits, M, K, N, sms) ? align16((size_t)codes_pitch(M) * K) : 0;
    return codes + (layer_forward_needs_sums(bits, M, K, N, sms) ? (size_t)M * N * sizeof(uint32_t) : 0);
}
static size_t layer_forward_rows_bytes(int M, int K, int N, int sms) {
    return align16((size_t)codes_pitch(M) * K) + (lutgemm::forward_rows_cut(M, K, N, sms) ? (size_t)M * N * sizeof(uint32_t) : 0);
}

static size_t layer_forward_scratch_bytes(int bits, int M, int K, int N) {
    if (!lutgemm::bits_supported(bits) || M <= 0 || K <= 0 || N <= 0) return 0;
    const int sms = current_num_sms();
    if (sms <= 0) return 0;
    const size_t base = layer_forward_base_bytes(bits, M, K, N, sms);
    const size_t rows = forward_by_rows(bits, M, K, N, sms) ? layer_forward_rows_bytes(M, K, N, sms) : 0;
    return base > rows ? base : rows;
}

static int layer_forward_impl(const uint8_t *a, const uint8_t *w, const uint16_t *lut, int bits, int M, int K, int N,
                              const lutgemm::ConvGeom &conv, const lutgemm::LayerEpilogue &e, void *scratch,
                              size_t scratch_bytes, void *stream) {
    if (!lutgemm::bits_supported(bits)) return LUTGEMM_E_BITS;
    if (M <= 0 || K <= 0 || N <= 0 || (reinterpret_cast<uintptr_t>(lut) & 1) || (reinterpret_cast<uintptr_t>(scratch) & 15))
        return LUTGEMM_E_BADARG;
    const int sms = current_num_sms();
    if (sms <= 0) return LUTGEMM_E_CUDA;
    const size_t given = scratch ? scratch_bytes : 0, codes = (size_t)codes_pitch(M) * K;
    const bool by_rows = forward_by_rows(bits, M, K, N, sms) && given >= layer_forward_rows_bytes(M, K, N, sms);
    if (by_rows ? !lutgemm::forward_rows_cut(M, K, N, sms) : !layer_forward_needs_sums(bits, M, K, N, sms))
        return forward_impl(a, w, nullptr, lut, bits, M, K, N, conv, scratch, scratch_bytes, stream, &e, by_rows);
    if (given < (by_rows ? layer_forward_rows_bytes(M, K, N, sms) : layer_forward_base_bytes(bits, M, K, N, sms))) {
        if (small_workspace_refused(M, N)) return LUTGEMM_E_SCRATCH;
        return lutgemm::forward_rowbcast(a, w, nullptr, lut, bits, M, K, N, conv, &e, sms, static_cast<cudaStream_t>(stream));
    }
    uint32_t *sums = reinterpret_cast<uint32_t *>(static_cast<char *>(scratch) + align16(codes));
    const int rc = forward_impl(a, w, sums, lut, bits, M, K, N, conv, scratch, codes, stream, nullptr, by_rows);
    if (rc != LUTGEMM_OK) return rc;
    return lutgemm::conv_epilogue(sums, e.box, e.sumw_t, e.taps, e.s_a, e.s_w, e.z_a, e.z_w, e.bias, e.out, M, e.L, N, sms,
                                  static_cast<cudaStream_t>(stream));
}

size_t lutgemm_conv2d_forward_layer_scratch_bytes(int bits, int B, int C, int H, int W, int Cout, int kh, int kw,
                                                  int stride, int pad, int dil) {
    lutgemm::ConvGeom g{};
    if (make_geom(B, C, H, W, kh, kw, stride, pad, dil, &g) != LUTGEMM_OK) return 0;
    return layer_forward_scratch_bytes(bits, B * g.Ho * g.Wo, C * kh * kw, Cout);
}

size_t lutgemm_forward_layer_scratch_bytes(int bits, int M, int K, int N) {
    return layer_forward_scratch_bytes(bits, M, K, N);
}

int lutgemm_conv2d_forward_layer(const uint8_t *x, const uint8_t *wmat, const uint16_t *lut, int bits, int B, int C, int H,
                                 int W, int Cout, int kh, int kw, int stride, int pad, int dil, const float *box,
                                 const float *sumw_t, const float *taps, const float *s_a, const float *s_w,
                                 const float *z_a, const float *z_w, const float *bias, float *out, void *scratch,
                                 size_t scratch_bytes, void *stream) {
    lutgemm::ConvGeom g{};
    int rc = make_geom(B, C, H, W, kh, kw, stride, pad, dil, &g);
    if (rc != LUTGEMM_OK) return rc;
    if (!x || !wmat || !lut || Cout <= 0) return LUTGEMM_E_BADARG;
    lutgemm::LayerEpilogue e{};
    rc = make_epilogue(box, sumw_t, taps, s_a, s_w, z_a, z_w, bias, out, g.Ho * g.Wo, &e);
    if (rc != LUTGEMM_OK) return rc;
    return layer_forward_impl(x, wmat, lut, bits, B * g.Ho * g.Wo, C * kh * kw, Cout, g, e, scratch, scratch_bytes, stream);
}

int lutgemm_forward_layer(const uint8_t *a, const uint8_t *w, const uint16_t *lut, int bits, int M, int K, int N,
                          const float *box, const float *sumw_t, const float *taps, const float *s_a, const float *s_w,
                          const float *z_a, const float *z_w, const float *bias, float *out, void *scratch,
                          size_t scratch_bytes, void *stream) {
    if (!a || !w || !lut) return LUTGEMM_E_BADARG;
    lutgemm::ConvGeom none{};
    lutgemm::LayerEpilogue e{};
    const int rc = make_epilogue(box, sumw_t, taps, s_a, s_w, z_a, z_w, bias, out, 1, &e);
    if (rc != LUTGEMM_OK) return rc;
    return layer_forward_impl(a, w, lut, bits, M, K, N, none, e, scratch, scratch_bytes, stream);
}

// ---- layer prologue / epilogue ---------------------------------------------------------------------------
int lutgemm_quantize_activations(const float *x, long stride_b, long stride_c, long stride_h, long stride_w, int B,
                                 int C, int H, int W, const float *scale, const float *zp_neg, float qmax,
                                 uint8_t *codes, float *chansum, void *stream) {
    if (!x || !scale || !zp_neg || !codes || B <= 0 || C <= 0 || H <= 0 || W <= 0 || !(qmax >= 1.f && qmax <= 255.f))
        return LUTGEMM_E_BADARG;
    const int sms = current_num_sms();
    if (sms <= 0) return LUTGEMM_E_CUDA;
    return lutgemm::quantize_codes(x, stride_b, stride_c, stride_h, stride_w, B, C, H, W, scale, zp_neg, qmax, codes,
                                   chansum, sms, static_cast<cudaStream_t>(stream));
}

int lutgemm_quantize_activations_backward(const float *x, long stride_b, long stride_c, long stride_h, long stride_w,
                                          int B, int C, int H, int W, const float *scale, const float *zp_neg,
                                          float qmax, const float *gcodes, const float *box_t, const float *s_w,
                                          const float *z_w, float *gx, void *stream) {
    if (!x || !scale || !zp_neg || !gcodes || !s_w || !z_w || !gx || B <= 0 || C <= 0 || H <= 0 || W <= 0)
        return LUTGEMM_E_BADARG;
    const int sms = current_num_sms();
    if (sms <= 0) return LUTGEMM_E_CUDA;
    return lutgemm::quantize_backward(x, stride_b, stride_c, stride_h, stride_w, B, C, H, W, scale, zp_neg, qmax, gcodes,
                                      box_t, s_w, z_w, gx, sms, static_cast<cudaStream_t>(stream));
}

int lutgemm_conv2d_epilogue(const uint32_t *y, const float *box, const float *sumw_t, const float *taps,
                            const float *s_a, const float *s_w, const float *z_a, const float *z_w, const float *bias,
                            float *out, long M, int L, int Cout, void *stream) {
    if (!y || !box || !sumw_t || !taps || !s_a || !s_w || !z_a || !z_w || !out || M <= 0 || L <= 0 || Cout <= 0)
        return LUTGEMM_E_BADARG;
    const int sms = current_num_sms();
    if (sms <= 0) return LUTGEMM_E_CUDA;
    return lutgemm::conv_epilogue(y, box, sumw_t, taps, s_a, s_w, z_a, z_w, bias, out, M, L, Cout, sms,
                                  static_cast<cudaStream_t>(stream));
}

// ---- small kernels of the layer wiring -----------------------------------------------------------------------
int lutgemm_layer_update_ranges(const float *act_lo, const float *act_hi, const float *w_lo, const float *w_hi,
                                float *act_min, float *act_max, float *act_seen, float *w_min, float *w_max, float *w_seen,
                                float keep, float momentum, float a_qmax, float w_qmax, float eps, float *quant,
                                void *stream) {
    if (!act_lo || !act_hi || !w_lo || !w_hi || !act_min || !act_max || !act_seen || !w_min || !w_max || !w_seen || !quant)
        return LUTGEMM_E_BADARG;
    return lutgemm::layer_update_ranges(act_lo, act_hi, w_lo, w_hi, act_min, act_max, act_seen, w_min, w_max, w_seen, keep,
                                        momentum, a_qmax, w_qmax, eps, quant, static_cast<cudaStream_t>(stream));
}

int lutgemm_layer_weight_prep(const float *weight, long s_co, long s_c, long s_h, long s_w, int Cout, int Cin, int kh, int kw,
                              const float *quant, float qmax, uint8_t *wmat, float *wsum, void *stream) {
    if (!weight || !quant || !wmat || !wsum || Cout <= 0 || Cin <= 0 || kh <= 0 || kw <= 0 || kh * kw > 4096)
        return LUTGEMM_E_BADARG;
    return lutgemm::layer_weight_prep(weight, s_co, s_c, s_h, s_w, Cout, Cin, kh, kw, quant, qmax, wmat, wsum,
                                      static_cast<cudaStream_t>(stream));
}

int lutgemm_layer_cross_terms(const float *wsum, int Cout, int Cin, int H, int W, int kh, int kw, int stride, int pad,
                              int dil, float *sumw_t, float *taps, void *stream) {
    lutgemm::ConvGeom g{};
    const int rc = make_geom(1, Cin, H, W, kh, kw, stride, pad, dil, &g);
    if (rc != LUTGEMM_OK) return rc;
    if (!wsum || !sumw_t || !taps || Cout <= 0) return LUTGEMM_E_BADARG;
    const int sms = current_num_sms();
    if (sms <= 0) return LUTGEMM_E_CUDA;
    return lutgemm::layer_cross_terms(wsum, Cout, g, sumw_t, taps, sms, static_cast<cudaStream_t>(stream));
}

int lutgemm_layer_window_sum(const float *img, int B, int H, int W, int kh, int kw, int stride, int pad, int dil,
                             float *box, void *stream) {
    lutgemm::ConvGeom g{};
    const int rc = make_geom(B, 1, H, W, kh, kw, stride, pad, dil, &g);
    if (rc != LUTGEMM_OK) return rc;
    if (!img || !box) return LUTGEMM_E_BADARG;
    const int sms = current_num_sms();
    if (sms <= 0) return LUTGEMM_E_CUDA;
    return lutgemm::layer_window_sum(img, g, box, sms, static_cast<cudaStream_t>(stream));
}

int lutgemm_layer_window_sum_adjoint(const float *gsum, int B, int H, int W, int kh, int kw, int stride, int pad, int dil,
                                     float *out, void *stream) {
    lutgemm::ConvGeom g{};
    const int rc = make_geom(B, 1, H, W, kh, kw, stride, pad, dil, &g);
    if (rc != LUTGEMM_OK) return rc;
    if (!gsum || !out) return LUTGEMM_E_BADARG;
    const int sms = current_num_sms();
    if (sms <= 0) return LUTGEMM_E_CUDA;
    return lutgemm::layer_window_sum_adjoint(gsum, g, out, sms, static_cast<cudaStream_t>(stream));
}

int lutgemm_layer_row_sums(const float *g, long M, int N, float *sums, void *stream) {
    if (!g || !sums || M <= 0 || N <= 0) return LUTGEMM_E_BADARG;
    const int sms = current_num_sms();
    if (sms <= 0) return LUTGEMM_E_CUDA;
    return lutgemm::layer_row_sums(g, M, N, sums, sms, static_cast<cudaStream_t>(stream));
}

int lutgemm_layer_weight_grad(const float *gwmat, const float *tapg, const float *weight, long s_co, long s_c, long s_h,
                              long s_w, int Cout, int Cin, int kh, int kw, const float *quant, float qmax, float *gw,
                              void *stream) {
    if (!gwmat || !tapg || !weight || !quant || !gw || Cout <= 0 || Cin <= 0 || kh <= 0 || kw <= 0) return LUTGEMM_E_BADARG;
    const int sms = current_num_sms();
    if (sms <= 0) return LUTGEMM_E_CUDA;
    return lutgemm::layer_weight_grad_finish(gwmat, tapg, weight, s_co, s_c, s_h, s_w, Cout, Cin, kh, kw, quant, qmax, gw,
                                             sms, static_cast<cudaStream_t>(stream));
}

// ---- a convolution layer's forward pass in one call --------------------------------------------------------------
size_t lutgemm_conv2d_layer_work_floats(int B, int C, int H, int W, int Cout, int kh, int kw, int stride, int pad, int dil) {
    lutgemm::ConvGeom g{};
    if (Cout <= 0 || make_geom(B, C, H, W, kh, kw, stride, pad, dil, &g) != LUTGEMM_OK) return 0;
    const size_t L = (size_t)g.Ho * g.Wo;
    return (size_t)B * H * W + (size_t)Cout * kh * kw + L * Cout + L + B * L;
}

int lutgemm_conv2d_layer_pass(const float *x, long x_sb, long x_sc, long x_sh, long x_sw, const float *weight, long w_so,
                              long w_sc, long w_sh, long w_sw, const float *bias, const float *quant, float a_qmax,
                              float w_qmax, const uint16_t *lut, int bits, int B, int C, int H, int W, int Cout, int kh,
                              int kw, int stride, int pad, int dil, uint8_t *codes, uint8_t *wmat, float *out, float *work,
                              void *scratch, size_t scratch_bytes, void *stream) {
    lutgemm::ConvGeom g{};
    int rc = make_geom(B, C, H, W, kh, kw, stride, pad, dil, &g);
    if (rc != LUTGEMM_OK) return rc;
    // everything the steps below would refuse, before the first of them writes anything
    if (!lutgemm::bits_supported(bits)) return LUTGEMM_E_BITS;
    if (!x || !weight || !quant || !lut || !codes || !wmat || !out || !work || Cout <= 0 || kh * kw > 4096 ||
        !(a_qmax >= 1.f && a_qmax <= 255.f) || (reinterpret_cast<uintptr_t>(lut) & 1) || (reinterpret_cast<uintptr_t>(out) & 3) ||
        (reinterpret_cast<uintptr_t>(work) & 3) || (reinterpret_cast<uintptr_t>(scratch) & 15))
        return LUTGEMM_E_BADARG;
    if (H > 65535 || B > 65535) return LUTGEMM_E_TOOLARGE;
    const int sms = current_num_sms(), M = B * g.Ho * g.Wo, K = C * kh * kw;
    if (sms <= 0) return LUTGEMM_E_CUDA;
    // (a buffer for codes and sums is enough for every choice; what the choice needs is only worked out for a smaller one)
    if (scratch_bytes < (size_t)codes_pitch(M) * K + (size_t)M * Cout * sizeof(uint32_t) && small_workspace_refused(M, Cout) &&
        scratch_bytes < layer_forward_base_bytes(bits, M, K, Cout, sms) && (scratch || layer_forward_needs_sums(bits, M, K, Cout, sms)))
        return LUTGEMM_E_SCRATCH;
    const size_t L = (size_t)g.Ho * g.Wo, pixels = (size_t)B * H * W;
    float *chansum = work, *wsum = chansum + pixels, *sumw_t = wsum + (size_t)Cout * kh * kw, *taps = sumw_t + L * Cout,
          *box = taps + L;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    rc = lutgemm::layer_prep(x, x_sb, x_sc, x_sh, x_sw, B, C, H, W, a_qmax, weight, w_so, w_sc, w_sh, w_sw, Cout, kh, kw, w_qmax, quant,
                             codes, chansum, wmat, wsum, sms, s);
    if (rc == LUTGEMM_OK) rc = lutgemm::layer_sums(wsum, Cout, g, sumw_t, taps, chansum, box, sms, s);
    if (rc != LUTGEMM_OK) return rc;
    return lutgemm_conv2d_forward_layer(codes, wmat, lut, bits, B, C, H, W, Cout, kh, kw, stride, pad, dil, box, sumw_t, taps,
                                        quant, quant + 2, quant + 1, quant + 3, bias, out, scratch, scratch_bytes, stream);
}

}  // extern "C"
