"""GPU tests of the gradient kernel with one thread per output row (512 rows x 64 terms) at the sizes where it can go wrong:
remainders of its row tiles, term blocks, slab buffers and 16-k operand stages, sums over several groups and over runs of
term blocks, stride classes and pointwise windows, with tables over the whole int16 range.

Tolerance: as for the other gradient kernels, 1e-5 of the sum of the absolute terms.  The longest chain of additions here is
16 terms in a thread, 16 blocks (or 8 blocks of a run and one addition per run) and the groups: fewer than 100, 6e-6."""
import numpy as np
import pytest
import torch

from oracle import oracle_np as O
from test_gpu_packed_slab import backward, check, full_range_tables, problem

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.fail("gpu-marked test started without a CUDA device")
    import approx_ops
    approx_ops.library()
    return torch.device("cuda:0")


@pytest.fixture
def rows():
    import approx_ops
    approx_ops.set_kernel_choice(backward="slab", grad_tile="rows")
    yield
    approx_ops.set_kernel_choice()


def slope_tables(bits, seed, least):
    """Entries from `least` up to 2040, as slopes of products have them."""
    rng = np.random.default_rng(seed)
    q = 1 << bits
    out = []
    for _ in range(2):
        t = rng.integers(least, 2041, (q, q))
        t[0, 0], t[q - 1, q - 1] = least, 2040
        out.append(O.pack_padded(t, bits, np.int16))
    return out


@pytest.mark.parametrize("table", ["full", "slopes"])
@pytest.mark.parametrize("bits", [4, 6, 7, 8])
@pytest.mark.parametrize("M,K,N", [(511, 1, 65), (512, 2, 64), (513, 3, 63), (70, 15, 513), (530, 16, 130), (40, 17, 1030),
                                   (33, 33, 1100), (600, 47, 66), (1500, 150, 20), (20000, 9, 12)])
def test_gradients_at_the_edges_of_tiles_blocks_and_stages(dev, oracle_c, rows, bits, M, K, N, table):
    la, lw = full_range_tables(bits, 3 * bits) if table == "full" else slope_tables(bits, 3 * bits, -100)
    a, w, gc = problem(bits, M, K, N, bits + M + K + N)
    ga, gw = backward(dev, gc, a, w, la, lw)
    ga2, gw2 = backward(dev, gc, a, w, la, lw)
    assert np.array_equal(ga, ga2) and np.array_equal(gw, gw2)  # the order of the additions is fixed
    r_ga, r_gw, r_gaa, r_gwa = oracle_c.backward_f64(gc, a, w, la, lw, bits)
    check(ga, r_ga, r_gaa)
    check(gw, r_gw, r_gwa)


@pytest.mark.parametrize("bits,M,K,N", [(4, 40000, 1500, 20), (7, 40000, 1500, 20), (8, 40000, 1500, 20), (7, 300, 300, 8200),
                                        (8, 300, 300, 8200)])
def test_long_sums(dev, oracle_c, rows, bits, M, K, N):
    """Runs of term blocks through the CTA's buffer (625 and 129 blocks of terms), whole rounds and a last one with K cut."""
    la, lw = full_range_tables(bits, 11 * bits)
    a, w, gc = problem(bits, M, K, N, bits + M)
    ga, gw = backward(dev, gc, a, w, la, lw)
    r_ga, r_gw, r_gaa, r_gwa = oracle_c.backward_f64(gc, a, w, la, lw, bits)
    check(ga, r_ga, r_gaa)
    check(gw, r_gw, r_gwa)


@pytest.mark.parametrize("least", [0, -100, -510, -511])
@pytest.mark.parametrize("scale", [1.0, 1e-17, 1e17, 1e-19, 1e19, 1e-37, 1e33])
def test_grad_out_of_any_size(dev, oracle_c, rows, least, scale):
    """Values near both ends of the fp32 range, and tables that reach below zero by a quarter of their largest entry."""
    bits, M, K, N = 7, 530, 20, 200
    la, lw = slope_tables(bits, 5, least)
    a, w, gc = problem(bits, M, K, N, 3)
    gc[: M // 2] = 0.0
    gc *= np.float32(scale)
    ga, gw = backward(dev, gc, a, w, la, lw)
    r_ga, r_gw, r_gaa, r_gwa = oracle_c.backward_f64(gc, a, w, la, lw, bits)
    check(ga, r_ga, r_gaa)
    check(gw, r_gw, r_gwa)


@pytest.mark.parametrize("least", [0, -100])
def test_infinities_and_nan_in_grad_out(dev, least):
    """They end up where the kernels with terms across lanes put them (0 * inf among the products)."""
    import approx_ops
    bits, M, K, N = 7, 600, 20, 200
    la, lw = slope_tables(bits, 5, least)
    a, w, gc = problem(bits, M, K, N, 4)
    gc[3, 7], gc[100, 199], gc[599, 0], gc[599, 1] = np.inf, -np.inf, np.nan, 3e38
    t = [torch.from_numpy(x).to(dev) for x in (gc, a, w, la, lw)]
    out = []
    try:
        for tile in ("wide", "rows"):
            approx_ops.set_kernel_choice(backward="slab", grad_tile=tile)
            ga, gw = torch.zeros(a.shape, device=dev), torch.zeros(w.shape, device=dev)
            approx_ops.approx_gemm_backward(t[0], t[1], t[2], ga, gw, t[3], t[4])
            out.append((ga, gw))
    finally:
        approx_ops.set_kernel_choice()
    for x, y in zip(*out):
        assert not torch.isfinite(x).all()
        assert torch.equal(torch.isnan(x), torch.isnan(y)) and torch.equal(torch.isinf(x), torch.isinf(y))
        assert torch.equal(torch.sign(x[torch.isinf(x)]), torch.sign(y[torch.isinf(y)]))


@pytest.mark.parametrize("bits", [4, 6, 7, 8])
@pytest.mark.parametrize("B,Cin,H,Cout,k,st,p", [(1, 5, 9, 64, 3, 1, 1), (2, 33, 6, 128, 3, 1, 1), (1, 18, 7, 63, 3, 1, 1), (2, 9, 7, 2, 3, 1, 1),
                                                 (1, 16, 9, 256, 3, 2, 1), (37, 20, 16, 128, 3, 1, 1), (4, 18, 40, 20, 5, 3, 2),
                                                 (3, 40, 13, 72, 1, 1, 0), (3, 40, 13, 72, 1, 2, 0)])
def test_image_gradient_of_convolutions(dev, oracle_c, rows, bits, B, Cin, H, Cout, k, st, p):
    import approx_ops
    la, lw = slope_tables(bits, 5 * bits, -100)
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
    assert approx_ops.device_error() == 0
    r_ga, r_gw, r_gaa, r_gwa = oracle_c.backward_f64(gy, col, wmat, la, lw, bits)
    check(gw.cpu().numpy(), r_gw, r_gwa)
    check(gx.cpu().numpy(), O.col2im_f64(r_ga, x.shape, k, k, st, p, 1), O.col2im_f64(r_gaa, x.shape, k, k, st, p, 1))
