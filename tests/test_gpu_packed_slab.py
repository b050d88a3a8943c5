"""GPU tests of the packed-slab gradient kernels (512 x 64 tiles, 576 x 64 for grad_x) at the sizes where they can go
wrong - remainders of tiles, of the two-k slab buffers and of the 16-k operand stages - with tables over the whole int16
range, of the forward kernel's two-k pipeline, and of what the dispatcher does when a caller's scratch buffer is too small
for the faster kernel.

Tolerance: an fp32 sum of n terms in any order is off by at most about n * 2^-24 times the sum of the absolute terms, and
the kernels add at most 16 terms per accumulator, 32 accumulators and the row blocks in turn (fewer than 100 additions in
a chain, 6e-6); 1e-5 of the sum of the absolute terms is what every gradient test here allows."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import oracle_np as O

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.fail("gpu-marked test started without a CUDA device")
    import approx_ops
    approx_ops.library()
    return torch.device("cuda:0")


@pytest.fixture
def packed():
    import approx_ops
    approx_ops.set_kernel_choice(backward="slab", grad_tile="wide")
    yield
    approx_ops.set_kernel_choice()


def full_range_tables(bits, seed):
    rng = np.random.default_rng(seed)
    q = 1 << bits
    out = []
    for _ in range(2):
        t = rng.integers(-2 ** 15, 2 ** 15, (q, q))
        t[0, 0], t[q - 1, q - 1], t[0, q - 1], t[q - 1, 0] = -2 ** 15, 2 ** 15 - 1, 0, -1
        out.append(O.pack_padded(t, bits, np.int16))
    return out


def problem(bits, M, K, N, seed):
    rng = np.random.default_rng(seed)
    q = 1 << bits
    a, w = rng.integers(0, q, (M, K)).astype(np.uint8), rng.integers(0, q, (K, N)).astype(np.uint8)
    return a, w, rng.standard_normal((M, N)).astype(np.float32)


def backward(dev, gc, a, w, la, lw):
    import approx_ops
    ga = torch.full(a.shape, float("nan"), dtype=torch.float32, device=dev)
    gw = torch.full(w.shape, float("nan"), dtype=torch.float32, device=dev)
    t = [torch.from_numpy(x).to(dev) for x in (gc, a, w, la, lw)]
    approx_ops.approx_gemm_backward(t[0], t[1], t[2], ga, gw, t[3], t[4])
    torch.cuda.synchronize()
    assert approx_ops.device_error() == 0
    return ga.cpu().numpy(), gw.cpu().numpy()


def check(got, ref, refabs):
    assert np.isfinite(got).all()
    assert (np.abs(got - ref) <= TOL * refabs + 1e-30).all()


@pytest.mark.parametrize("bits", [4, 6, 7, 8])
@pytest.mark.parametrize("M,K,N", [(511, 1, 65), (512, 2, 64), (513, 3, 63), (70, 15, 513), (530, 16, 130), (1030, 17, 40),
                                   (33, 33, 1100), (600, 47, 66), (20000, 9, 12), (20000, 7, 5)])
def test_gradients_at_the_edges_of_tiles_and_stages(dev, oracle_c, packed, bits, M, K, N):
    """(The last two have 40 row blocks: the many-block reduction with and without 16-byte vectors.)"""
    la, lw = full_range_tables(bits, 3 * bits)
    a, w, gc = problem(bits, M, K, N, bits + M + K + N)
    ga, gw = backward(dev, gc, a, w, la, lw)
    r_ga, r_gw, r_gaa, r_gwa = oracle_c.backward_f64(gc, a, w, la, lw, bits)
    check(ga, r_ga, r_gaa)
    check(gw, r_gw, r_gwa)


@pytest.mark.parametrize("bits,M,K,N", [(4, 130300, 33, 20), (6, 130300, 33, 20), (7, 130300, 33, 20), (8, 130300, 33, 20),
                                        (7, 11015, 66, 700), (8, 11015, 66, 700)])
def test_gradients_with_several_row_blocks_per_cta(dev, oracle_c, packed, bits, M, K, N):
    """grad_w with two row blocks added up in each of 128 groups, the last one short; grad_a with both of its row blocks added up,
    whole rounds of tiles and a last round with K cut.  The order of the additions is fixed: a second run is identical."""
    la, lw = full_range_tables(bits, 11 * bits)
    a, w, gc = problem(bits, M, K, N, bits + M)
    ga, gw = backward(dev, gc, a, w, la, lw)
    ga2, gw2 = backward(dev, gc, a, w, la, lw)
    assert np.array_equal(ga, ga2) and np.array_equal(gw, gw2)
    r_ga, r_gw, r_gaa, r_gwa = oracle_c.backward_f64(gc, a, w, la, lw, bits)
    check(ga, r_ga, r_gaa)
    check(gw, r_gw, r_gwa)


@pytest.mark.parametrize("bits", [4, 6, 7, 8])
@pytest.mark.parametrize("B,Cin,H,Cout,k,st,p", [(1, 5, 9, 64, 3, 1, 1), (2, 33, 6, 128, 3, 1, 1), (1, 18, 7, 63, 3, 1, 1),
                                                 (1, 16, 9, 256, 3, 2, 1), (37, 20, 16, 128, 3, 1, 1), (4, 18, 40, 128, 3, 1, 1)])
def test_image_gradient_of_convolutions(dev, oracle_c, packed, bits, B, Cin, H, Cout, k, st, p):
    """576-row tiles (one and two of them, and a partly filled one), the stride classes of a stride-2 convolution; 148 pixel
    tiles whose two row blocks one CTA adds up, and more work items than SMs, so that a CTA takes a second one."""
    import approx_ops
    la, lw = full_range_tables(bits, 5 * bits)
    rng = np.random.default_rng(bits + Cin + Cout)
    q = 1 << bits
    x = rng.integers(0, q, (B, Cin, H, H)).astype(np.uint8)
    wmat = rng.integers(0, q, (Cin * k * k, Cout)).astype(np.uint8)
    Ho = (H + 2 * p - k) // st + 1
    gy = rng.standard_normal((B * Ho * Ho, Cout)).astype(np.float32)
    col = oracle_c.im2col(x, k, k, st, p, 1)
    gx = torch.full(x.shape, float("nan"), dtype=torch.float32, device=dev)
    gw = torch.full(wmat.shape, float("nan"), dtype=torch.float32, device=dev)
    t = [torch.from_numpy(v).to(dev) for v in (gy, x, wmat, la, lw)]
    approx_ops.approx_conv2d_backward(t[0], t[1], t[2], gx, gw, t[3], t[4], k, k, st, p, 1)
    r_ga, r_gw, r_gaa, r_gwa = oracle_c.backward_f64(gy, col, wmat, la, lw, bits)
    check(gw.cpu().numpy(), r_gw, r_gwa)
    check(gx.cpu().numpy(), O.col2im_f64(r_ga, x.shape, k, k, st, p, 1), O.col2im_f64(r_gaa, x.shape, k, k, st, p, 1))


@pytest.mark.parametrize("bits", [6, 7, 8])
def test_a_small_scratch_buffer_selects_a_kernel_that_fits(dev, oracle_c, bits):
    """A buffer that the choice by fixed limits can work with is not refused: the gradients are then computed by its
    kernels.  Without a buffer the broadcast kernels, which need none here, run."""
    import approx_ops
    lib = approx_ops.library()
    la, lw = full_range_tables(bits, 7 * bits)
    M, K, N = 300, 200, 600  # slab kernels by estimated time; M < 512 and N < 768: broadcast kernels by fixed limits
    a, w, gc = problem(bits, M, K, N, bits)
    assert lib.lutgemm_backward_scratch_bytes(bits, M, K, N) > 0
    ga, gw = (torch.full(s, float("nan"), dtype=torch.float32, device=dev) for s in (a.shape, w.shape))
    t = [torch.from_numpy(v).to(dev) for v in (gc, a, w, la, lw)]
    rc = lib.lutgemm_backward(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), ga.data_ptr(), gw.data_ptr(), t[3].data_ptr(),
                              t[4].data_ptr(), bits, M, K, N, None, 0, None)
    assert rc == 0
    torch.cuda.synchronize()
    r_ga, r_gw, r_gaa, r_gwa = oracle_c.backward_f64(gc, a, w, la, lw, bits)
    check(ga.cpu().numpy(), r_ga, r_gaa)
    check(gw.cpu().numpy(), r_gw, r_gwa)
    # 4096 rows, the weight gradient by a slab kernel under either choice: a buffer below both needs is refused (the
    # buffers have their full sizes, so that a call that were accepted would stay inside them)
    if bits >= 7:
        a, w, gc = problem(bits, 4096, K, N, bits)
        t = [torch.from_numpy(v).to(dev) for v in (gc, a, w, la, lw)]
        ga, gw = (torch.zeros(s, dtype=torch.float32, device=dev) for s in (a.shape, w.shape))
        scratch = torch.empty(lib.lutgemm_backward_scratch_bytes(bits, 4096, K, N), dtype=torch.uint8, device=dev)
        launches = lib.lutgemm_kernel_launches()
        rc = lib.lutgemm_backward(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), ga.data_ptr(), gw.data_ptr(), t[3].data_ptr(),
                                  t[4].data_ptr(), bits, 4096, K, N, scratch.data_ptr(), 16, None)
        assert rc == -4 and lib.lutgemm_kernel_launches() == launches  # LUTGEMM_E_SCRATCH, before anything is launched


@pytest.mark.parametrize("bits", [6, 7, 8])
def test_image_gradient_without_scratch(dev, oracle_c, bits):
    import approx_ops
    lib = approx_ops.library()
    la, lw = full_range_tables(bits, 9 * bits)
    B, Cin, H, Cout, k = 1, 64, 8, 256, 3
    assert lib.lutgemm_conv2d_backward_scratch_bytes(bits, B, Cin, H, H, Cout, k, k, 1, 1, 1) > 0
    rng = np.random.default_rng(bits)
    x = rng.integers(0, 1 << bits, (B, Cin, H, H)).astype(np.uint8)
    wmat = rng.integers(0, 1 << bits, (Cin * k * k, Cout)).astype(np.uint8)
    gy = rng.standard_normal((B * H * H, Cout)).astype(np.float32)
    gx = torch.full(x.shape, float("nan"), dtype=torch.float32, device=dev)
    t = [torch.from_numpy(v).to(dev) for v in (gy, x, wmat, la)]
    rc = lib.lutgemm_conv2d_backward(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), gx.data_ptr(), None, t[3].data_ptr(), None,
                                     bits, B, Cin, H, H, Cout, k, k, 1, 1, 1, ctypes.c_void_p(None), 0, None)
    assert rc == 0
    torch.cuda.synchronize()
    col = oracle_c.im2col(x, k, k, 1, 1, 1)
    r_ga, _, r_gaa, _ = oracle_c.backward_f64(gy, col, wmat, la, lw, bits)
    check(gx.cpu().numpy(), O.col2im_f64(r_ga, x.shape, k, k, 1, 1, 1), O.col2im_f64(r_gaa, x.shape, k, k, 1, 1, 1))
    # it is the broadcast kernel that ran, and a slab kernel that would have (their sums differ in the last bits)
    other = {}
    try:
        for family in ("bcast", "auto"):
            approx_ops.set_kernel_choice(backward=family)
            other[family] = torch.empty_like(gx)
            approx_ops.approx_conv2d_backward(t[0], t[1], t[2], other[family], None, t[3], t[3], k, k, 1, 1, 1)
    finally:
        approx_ops.set_kernel_choice()
    assert torch.equal(gx, other["bcast"]) and not torch.equal(gx, other["auto"])


@pytest.mark.parametrize("bits", [4, 6, 7, 8])
@pytest.mark.parametrize("M,K,N", [(512, 80, 64), (700, 77, 90), (40, 301, 33), (512 * 296 - 100, 70, 20)])
def test_forward_slab_kernel_without_and_with_a_workspace(dev, bits, M, K, N):
    """Five and more 16-k operand chunks, a last one of 6, 13 or 16 k, tiles cut across CTAs and (the last) whole tiles of
    which a CTA takes two, with the three ways to stage operands: whole numbers, so equal to the broadcast kernel's sums."""
    import approx_ops
    lib = approx_ops.library()
    a, w, _ = problem(bits, M, K, N, bits + M)
    lut = O.pack_padded(np.random.default_rng(bits).integers(0, 2 ** 16, (1 << bits, 1 << bits)), bits, np.uint16)
    a, w, lut = (torch.from_numpy(v).to(dev) for v in (a, w, lut))
    out = []

    def run(family, ws, tma):
        approx_ops.set_kernel_choice(forward=family)
        lib.lutgemm_set_tma(tma)
        nbytes = lib.lutgemm_forward_scratch_bytes(bits, M, K, N) if ws else 0
        scratch = torch.empty(nbytes, dtype=torch.uint8, device=dev) if nbytes else None
        c = torch.full((M, N), 7, dtype=torch.int32, device=dev).view(torch.uint32)
        assert lib.lutgemm_forward_ws(a.data_ptr(), w.data_ptr(), c.data_ptr(), lut.data_ptr(), bits, M, K, N,
                                      scratch.data_ptr() if nbytes else None, nbytes, None) == 0
        torch.cuda.synchronize()
        out.append(c.view(torch.int32))
    try:
        run("rowbcast", False, 1)
        run("slab", False, 1)
        run("slab", True, 0)
        run("slab", True, 1)
    finally:
        approx_ops.set_kernel_choice()
        lib.lutgemm_set_tma(1)
    assert approx_ops.device_error() == 0
    assert all(torch.equal(out[0], o) for o in out[1:])


@pytest.mark.parametrize("M,K,N", [(256, 576, 64), (300, 200, 600), (40000, 100, 24)])
def test_forward_with_a_workspace_that_is_too_small(dev, M, K, N):
    """Shapes where only the estimate picks the slab kernel: sums and layer outputs are those of the full workspace."""
    import approx_ops
    lib, bits = approx_ops.library(), 7
    a, w, _ = problem(bits, M, K, N, M)
    lut = O.pack_padded(np.random.default_rng(2).integers(0, 2 ** 14, (128, 128)), bits, np.uint16)
    a, w, lut = (torch.from_numpy(v).to(dev) for v in (a, w, lut))
    box, sumw, taps = a.sum(dim=1, dtype=torch.float32), w.sum(dim=0, dtype=torch.float32), torch.full((1,), float(K), device=dev)
    q = torch.tensor([0.01, -3.0, 0.02, -60.0], device=dev)
    full = lib.lutgemm_forward_scratch_bytes(bits, M, K, N)
    full_layer = lib.lutgemm_forward_layer_scratch_bytes(bits, M, K, N)
    assert full > 64 and full_layer > 64
    scratch = torch.empty(max(full, full_layer), dtype=torch.uint8, device=dev)
    c, o = [], []
    for small in (False, True):
        c.append(torch.zeros((M, N), dtype=torch.int32, device=dev))
        o.append(torch.zeros((M, N), device=dev))
        assert lib.lutgemm_forward_ws(a.data_ptr(), w.data_ptr(), c[-1].data_ptr(), lut.data_ptr(), bits, M, K, N,
                                      scratch.data_ptr(), 64 if small else full, None) == 0
        assert lib.lutgemm_forward_layer(a.data_ptr(), w.data_ptr(), lut.data_ptr(), bits, M, K, N, box.data_ptr(), sumw.data_ptr(),
                                         taps.data_ptr(), q.data_ptr(), q[2:].data_ptr(), q[1:].data_ptr(), q[3:].data_ptr(), None,
                                         o[-1].data_ptr(), scratch.data_ptr(), 64 if small else full_layer, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(c[0], c[1]) and torch.equal(o[0], o[1])


@pytest.mark.parametrize("Cout,Cin,k", [(8, 5, 1), (13, 700, 1), (64, 33, 3), (9, 3, 23), (1, 1, 1)])
def test_weight_codes_and_their_sums(dev, Cout, Cin, k):
    """Eight channels per block with and without whole 8-byte stores, one tap, more taps than eight channels' sums fit
    shared memory, K below a warp and above a block: codes and sums are whole numbers, so the comparison is exact."""
    import approx_ops
    g = torch.Generator().manual_seed(Cout + Cin + k)
    w = torch.randn(Cout, Cin, k, k, generator=g)
    s, z, qmax = 0.0371, -31.0, 127.0
    quant = torch.tensor([1.0, 0.0, s, z], device=dev)
    for weight in (w.to(dev), w.to(dev).to(memory_format=torch.channels_last)):
        wmat, wsum = approx_ops.layer_weight_prep(weight, quant, qmax)
        codes = torch.clamp(torch.round(w / quant[2].cpu() - quant[3].cpu()), 0, qmax)
        assert torch.equal(wmat.cpu().float(), codes.reshape(Cout, -1).t())
        assert torch.equal(wsum.cpu(), codes.reshape(Cout, Cin, k * k).sum(dim=1))


@pytest.mark.parametrize("K", [2200001, 4200000])
def test_forward_over_a_long_k(dev, K):
    """The transposed code copy of the slab kernel in more than one launch (byte loads, and 16-byte loads through a tile):
    whole numbers, so equal to the broadcast kernel's sums, which need no copy."""
    import approx_ops
    M, N, bits = 16, 20, 4
    g = torch.Generator(device=dev).manual_seed(K)
    a = torch.randint(0, 16, (M, K), generator=g, device=dev, dtype=torch.uint8)
    w = torch.randint(0, 16, (K, N), generator=g, device=dev, dtype=torch.uint8)
    lut = torch.from_numpy(O.pack_padded(np.random.default_rng(1).integers(0, 2 ** 16, (16, 16)), bits, np.uint16)).to(dev)
    out = []
    try:
        for family in ("slab", "rowbcast"):
            approx_ops.set_kernel_choice(forward=family)
            out.append(torch.zeros((M, N), dtype=torch.uint32, device=dev))
            approx_ops.approx_gemm_forward(a, w, out[-1], lut)
    finally:
        approx_ops.set_kernel_choice()
    assert torch.equal(out[0].view(torch.int32), out[1].view(torch.int32))
