"""GPU tests of the one-pass kernels around the LUT kernels at the sizes where their tiles, vectors and layouts change: the
quantisation in channels-last and in flat order, the transposed code copy of convolutions, the de-quantisation four channels at a
time.  Codes, copies and window sums are whole numbers and compared for equality; gradients and outputs are the same
roundings in the same order as the reference expressions evaluated in fp32."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.fail("gpu-marked test started without a CUDA device")
    import approx_ops
    approx_ops.library()
    return torch.device("cuda:0")


@pytest.mark.parametrize("channels_last", [False, True])
@pytest.mark.parametrize("window", [False, True])
@pytest.mark.parametrize("B,C,H,W", [(1, 4, 1, 1), (2, 64, 8, 8), (3, 68, 7, 7), (1, 132, 5, 13), (2, 60, 9, 16), (1, 3, 11, 6), (4, 256, 1, 3), (1, 40, 1, 384),
                                     (1, 7, 1, 48)])
def test_quantisation_and_its_gradient(dev, B, C, H, W, window, channels_last):
    import approx_ops
    gen = torch.Generator(device=dev).manual_seed(B * C + H + W)
    x = torch.randn(B, C, H, W, generator=gen, device=dev)
    gcodes = torch.randn(B, C, H, W, generator=gen, device=dev)
    box = torch.randn(B, H, W, generator=gen, device=dev) if window else None
    s_a, z_a, s_w, z_w, qmax = (torch.tensor([v], device=dev) for v in (0.03, -40.0, 0.7, -55.0, 127.0))
    if channels_last:
        x = x.contiguous(memory_format=torch.channels_last)
    codes, chansum = approx_ops.quantize_activations(x, s_a, z_a, 127.0, want_chansum=window)
    q = torch.round(x / s_a - z_a)
    want = torch.clamp(q, 0, 127.0)
    assert torch.equal(codes.float(), want)
    assert chansum is None or torch.equal(chansum, want.sum(dim=1))
    gx = approx_ops.quantize_activations_backward(x, s_a, z_a, 127.0, gcodes, box, s_w, z_w)
    g = gcodes + z_w * box.unsqueeze(1) if window else gcodes
    mask = ((q >= 0) & (q <= 127.0)).float()
    assert gx.stride() == x.stride() and torch.equal(gx, mask * (s_w * g))


@pytest.mark.parametrize("B,C,H,W,k,s,p,d", [(3, 5, 8, 8, 3, 1, 1, 1), (70, 3, 4, 4, 3, 1, 1, 1), (2, 3, 32, 32, 3, 1, 1, 1), (2, 4, 16, 16, 3, 2, 1, 1), (5, 3, 8, 8, 1, 1, 0, 1),
                                             (3, 2, 9, 9, 1, 2, 0, 1), (2, 3, 16, 16, 1, 2, 0, 1), (2, 2, 30, 34, 5, 1, 1, 1), (1, 3, 24, 24, 3, 3, 1, 1),
                                             (2, 3, 20, 20, 3, 1, 2, 2), (2, 2, 19, 23, 7, 2, 3, 1), (1, 2, 8, 12, 3, 1, 0, 1), (3, 1, 64, 64, 3, 1, 1, 1)])
def test_transposed_codes_of_a_convolution(dev, B, C, H, W, k, s, p, d):
    """What the forward pass leaves for the backward pass: the unfolded codes, transposed."""
    import approx_ops
    gen = torch.Generator(device=dev).manual_seed(H * W + k)
    x = torch.randint(0, 128, (B, C, H, W), generator=gen, device=dev, dtype=torch.uint8)
    Cout = 40
    w = torch.randint(0, 128, (C * k * k, Cout), generator=gen, device=dev, dtype=torch.uint8)
    col = F.unfold(F.pad(x.float(), (p, p, p, p)), k, dilation=d, stride=s)  # [B, K, L]
    K, L = col.shape[1:]
    M, pitch = B * L, (B * L + 15) // 16 * 16
    want = torch.zeros(K, pitch, device=dev)
    want[:, :M] = col.permute(1, 0, 2).reshape(K, M)
    y = torch.empty(M, Cout, dtype=torch.int32, device=dev)
    lut = torch.zeros(approx_ops.library().lutgemm_lut_elem_num(7), dtype=torch.uint16, device=dev)
    try:
        approx_ops.set_kernel_choice(forward="slab")
        codes = approx_ops.approx_conv2d_forward(x, w, y.view(torch.uint32), lut, k, k, s, p, d)
    finally:
        approx_ops.set_kernel_choice()
    assert torch.equal(codes.view(K, pitch).float(), want)


@pytest.mark.parametrize("M,L,Cout", [(7, 7, 4), (30, 10, 68), (1000, 25, 64), (33, 11, 33), (5, 1, 1000)])
@pytest.mark.parametrize("with_bias", [False, True])
def test_dequantisation(dev, M, L, Cout, with_bias):
    import approx_ops
    gen = torch.Generator(device=dev).manual_seed(M + Cout)
    y = torch.randint(0, 2 ** 22, (M, Cout), generator=gen, device=dev, dtype=torch.int32)
    box, sumw, taps = (torch.randint(0, 3000, n, generator=gen, device=dev).float() for n in ((M,), (L, Cout), (L,)))
    s_a, s_w, z_a, z_w = (torch.tensor([v], device=dev) for v in (0.013, 0.021, -3.0, -61.0))
    bias = torch.randn(Cout, generator=gen, device=dev) if with_bias else None
    out = approx_ops.conv2d_epilogue(y.view(torch.uint32), box, sumw, taps, s_a, s_w, z_a, z_w, bias, L)
    l = torch.arange(M, device=dev) % L
    acc = y.float() + (z_w * box)[:, None] + z_a * sumw[l] + ((z_a * z_w) * taps[l])[:, None]
    want = (s_a * s_w) * acc
    assert torch.equal(out, want + bias if with_bias else want)


@pytest.mark.parametrize("B,C,H,W,Cout,k,s,p", [(2, 64, 8, 8, 64, 3, 1, 1), (1, 4, 1, 1, 8, 1, 1, 0), (3, 132, 7, 7, 20, 3, 2, 1), (1, 516, 3, 5, 9, 1, 1, 0), (40, 516, 14, 14, 16, 3, 1, 1),
                                                (2, 68, 9, 9, 40, 5, 1, 2), (2, 3, 9, 9, 24, 3, 1, 1), (1, 4, 30, 30, 8, 23, 1, 0)])
@pytest.mark.parametrize("channels_last", [False, True])
def test_prologue_of_a_layer_in_one_launch(dev, B, C, H, W, Cout, k, s, p, channels_last):
    """One call against the entry points that it joins: all of them whole numbers until the last, so the results are equal."""
    import approx_ops
    import self_ops
    from lutgemm_luts import synthetic_multiplier, window_difference_gradients
    from self_ops.ops_py import approx_ops as state
    fp = synthetic_multiplier(7, seed=0)
    self_ops.set_lookup_tables(dev, fp, *window_difference_gradients(fp, 8), 7)
    gen = torch.Generator(device=dev).manual_seed(C + Cout)
    fmt = torch.channels_last if channels_last else torch.contiguous_format
    x = torch.randn(B, C, H, W, generator=gen, device=dev).contiguous(memory_format=fmt)
    weight = torch.randn(Cout, C, k, k, generator=gen, device=dev).contiguous(memory_format=fmt)
    quant = torch.tensor([0.04, -50.0, 0.03, -61.0], device=dev)
    s_a, z_a, s_w, z_w = (quant[i:i + 1] for i in range(4))
    codes, chansum = approx_ops.quantize_activations(x, s_a, z_a, 127.0)
    wq = torch.clamp(torch.round(weight / s_w - z_w), 0, 127.0)
    wmat, wsum = approx_ops.layer_weight_prep(weight, quant, 127.0)
    assert torch.equal(wmat.float(), wq.reshape(Cout, -1).t()) and torch.equal(wsum.view(Cout, -1), wq.sum(dim=1).reshape(Cout, -1))
    sumw_t, taps = approx_ops.layer_cross_terms(wsum, C, H, W, k, k, s, p, 1)
    box = approx_ops.layer_window_sum(chansum, k, k, s, p, 1)
    out, _ = approx_ops.approx_conv2d_forward_layer(codes, wmat, state.lut_appmult, k, k, s, p, 1, box, sumw_t, taps, s_a, s_w, z_a, z_w, None)
    got = approx_ops.conv2d_layer_pass(x, weight, None, quant, 127.0, 127.0, state.lut_appmult, s, p, 1)
    assert torch.equal(got[0].reshape(out.shape), out) and torch.equal(got[1], codes) and torch.equal(got[2], wmat)


@pytest.mark.parametrize("M,N", [(1, 1), (3, 2), (7, 33), (1001, 5), (517, 4), (130, 8), (65, 60), (4099, 64), (33, 132), (5, 1536), (9, 777), (200000, 12)])
def test_row_sums(dev, M, N):
    """|error| <= (4 + ceil(N / 128) + 5) * 2^-24 * sum |g|: four values of a vector, a lane's vectors one after the other (single
    values where N is odd: ceil(N / 32) of them), five halvings of a warp."""
    import approx_ops
    g = torch.randn(M, N, generator=torch.Generator(device=dev).manual_seed(N), device=dev)
    want = g.double().sum(dim=1)
    bound = (9 + -(-N // 32)) * 2.0 ** -24 * g.double().abs().sum(dim=1)
    assert bool(((approx_ops.layer_row_sums(g).double() - want).abs() <= bound).all())


@pytest.mark.parametrize("B,C,H,W,k,s,p,d", [(2, 3, 24, 18, 3, 1, 1, 1), (70, 2, 8, 6, 3, 1, 1, 1), (3, 2, 48, 36, 3, 2, 1, 1), (2, 3, 16, 17, 3, 1, 1, 1),
                                             (2, 2, 16, 22, 5, 1, 2, 1), (5, 3, 8, 2, 1, 1, 0, 1), (3, 2, 16, 1, 3, 1, 1, 1), (2, 2, 48, 50, 3, 3, 0, 1),
                                             (2, 3, 18, 24, 3, 1, 2, 2), (1, 2, 64, 66, 7, 1, 3, 1)])
def test_transposed_codes_of_output_rows_that_are_no_multiple_of_four(dev, B, C, H, W, k, s, p, d):
    test_transposed_codes_of_a_convolution(dev, B, C, H, W, k, s, p, d)


@pytest.mark.parametrize("B,C,H,W,k,s,p,d", [(2, 2, 48, 48, 1, 3, 0, 1), (2, 3, 47, 35, 1, 2, 0, 1), (3, 2, 14, 14, 1, 2, 1, 1), (9, 3, 8, 8, 1, 2, 0, 1),
                                             (1, 2, 64, 64, 1, 4, 0, 1)])
def test_transposed_codes_of_windows_one_row_high(dev, B, C, H, W, k, s, p, d):
    test_transposed_codes_of_a_convolution(dev, B, C, H, W, k, s, p, d)
