"""GPU tests of the small one-pass kernels of the layer wiring (lutgemm_layer_aux.cu), called through the C-ABI via
`approx_ops`, each against the PyTorch expression it replaces in the layer - the expressions the reference's
ApproxConv2d and observers evaluate (micronet+/app_layers.py:21-53, 147-184).  Sums of integer codes are exact, so
those comparisons are bit-exact; the others allow fp32 rounding of one operation."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

GEOMS = [  # B, Cin, H, W, Cout, kh, kw, stride, pad, dil
    (2, 5, 9, 11, 7, 3, 3, 1, 1, 1), (3, 4, 12, 12, 6, 3, 3, 2, 1, 1), (1, 3, 10, 8, 4, 5, 5, 1, 2, 1),
    (2, 2, 13, 13, 3, 3, 3, 1, 2, 2), (2, 6, 8, 8, 5, 1, 1, 2, 0, 1), (1, 2, 7, 9, 3, 2, 2, 3, 0, 1)]


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available(), "gpu-marked test started without a CUDA device"
    import approx_ops
    approx_ops.library()
    return torch.device("cuda:0")


def test_observers_and_quantisation_parameters_in_one_launch(dev):
    """layer_update_ranges against the PyTorch observers of lutgemm_layers (running weight range, moving-average
    activation range, scales, zero points) over four steps: identical buffers."""
    import approx_ops
    from lutgemm_layers import AppConv2d
    torch.manual_seed(0)
    ref = AppConv2d(4, 6, 3, 1, 1, 1, 1, False, 7, 7, False, "fused").to(dev).train()
    new = AppConv2d(4, 6, 3, 1, 1, 1, 1, False, 7, 7, False, "layer").to(dev).train()
    new.load_state_dict(ref.state_dict())
    for step in range(4):
        x = torch.randn(2, 4, 8, 8, device=dev) * (1.0 + step) - 0.3 * step
        with torch.no_grad():
            ref.weight.add_(0.05 * torch.randn_like(ref.weight))
            new.weight.copy_(ref.weight)
        ref._refresh(x, ref.weight)
        new._refresh(x, new.weight, fused=True)
        assert torch.equal(ref.quant, new.quant), step
        for a_, b_ in zip(ref.act_range.state() + ref.weight_range.state(), new.act_range.state() + new.weight_range.state()):
            assert torch.equal(a_, b_), step


@pytest.mark.parametrize("channels_last", [False, True])
def test_weight_codes_and_cross_terms(dev, channels_last):
    import approx_ops
    from lutgemm_layers import _valid_taps
    for s_, (B, Cin, H, W, Cout, kh, kw, st, p, d) in enumerate(GEOMS):
        torch.manual_seed(s_)
        weight = torch.randn(Cout, Cin, kh, kw, device=dev)
        if channels_last:
            weight = weight.contiguous(memory_format=torch.channels_last)
        qmax = 127.0
        quant = torch.tensor([0.03, -20.0, 0.02, -70.0], device=dev)
        wmat, wsum = approx_ops.layer_weight_prep(weight, quant, qmax)
        qw = torch.clamp(torch.round(weight / quant[2] - quant[3]), 0.0, qmax)
        assert torch.equal(wmat, qw.reshape(Cout, -1).t().to(torch.uint8))
        assert torch.equal(wsum, qw.sum(dim=1).reshape(Cout, kh * kw))
        sumw_t, taps = approx_ops.layer_cross_terms(wsum, Cin, H, W, kh, kw, st, p, d)
        if kh == kw:
            valid = _valid_taps((H, W, kh, kw, st, p, d), dev)  # [kh*kw, L]
            assert torch.equal(sumw_t, valid.t() @ wsum.t())
            assert torch.equal(taps, valid.sum(dim=0) * float(Cin))
        # gradient of the fp32 weight from the gradient of its codes
        gwmat = torch.randn(Cin * kh * kw, Cout, device=dev)
        tapg = torch.randn(Cout, kh * kw, device=dev)
        gw = approx_ops.layer_weight_grad(gwmat, tapg, weight, quant, qmax)
        g_qw = gwmat.t().reshape(weight.shape) + quant[1] * tapg.reshape(Cout, 1, kh, kw)
        q = torch.round(weight / quant[2] - quant[3])
        want = torch.where((q >= 0) & (q <= qmax), quant[0] * g_qw, torch.zeros_like(g_qw))
        assert gw.is_contiguous() and torch.equal(gw, want.contiguous())


def test_window_sums(dev):
    import approx_ops
    from lutgemm_layers import _out_hw, _window_sum, _window_sum_adjoint
    for s_, (B, Cin, H, W, Cout, kh, kw, st, p, d) in enumerate(GEOMS):
        if kh != kw:
            continue
        torch.manual_seed(10 + s_)
        geom = (H, W, kh, kw, st, p, d)
        img = torch.randint(0, 128 * Cin, (B, H, W), device=dev).float()   # channel sums of codes: integers
        box = approx_ops.layer_window_sum(img, kh, kw, st, p, d)
        assert torch.equal(box, _window_sum(img, geom).reshape(-1))
        Ho, Wo = _out_hw(H, W, kh, kw, st, p, d)
        g = torch.randn(B, Ho, Wo, device=dev)
        adj = approx_ops.layer_window_sum_adjoint(g, H, W, kh, kw, st, p, d)
        want = _window_sum_adjoint(g, geom)
        assert torch.allclose(adj, want, rtol=0, atol=1e-6 * float(want.abs().max()))
        # <window_sum(u), g> = <u, adjoint(g)>
        u = torch.randn(B, H, W, device=dev)
        lhs = float((approx_ops.layer_window_sum(u, kh, kw, st, p, d).double() * g.reshape(-1).double()).sum())
        rhs = float((u.double() * adj.double()).sum())
        assert abs(lhs - rhs) <= 1e-5 * max(abs(lhs), 1.0)


def test_quantisation_division_matches_ieee_division_for_awkward_scales(dev):
    """The quantisation kernels divide by the common scale with a reciprocal and one fused correction; the codes must
    equal clamp(round(x / scale - zp)) evaluated with PyTorch's IEEE division for scales whose mantissa is all ones,
    a power of two, or random, and for activations that are zero, tiny, huge or infinite."""
    import approx_ops
    g = torch.Generator(device=dev).manual_seed(5)
    x = torch.randn(4, 40, 9, 33, device=dev, generator=g) * 3.0
    flat = x.view(-1)
    flat[::97] = 0.0
    flat[1::193] = 1e-38
    flat[2::211] = -3e37
    flat[3::389] = float("inf")
    flat[4::401] = -float("inf")
    x = x.contiguous(memory_format=torch.channels_last)
    mant = [0x7FFFFF, 0x7FFFFE, 0x000000, 0x000001, 0x400000, 0x2AAAAB, 0x555555, 0x123457]
    for bits, qmax in ((7, 127.0), (8, 255.0)):
        for i, m in enumerate(mant):
            for e in (110, 121, 127, 130):
                scale = torch.tensor([(e << 23) | m], dtype=torch.int32, device=dev).view(torch.float32)
                zp = torch.tensor([float(-(17 + 9 * i) % int(qmax))], device=dev).neg()
                codes, _ = approx_ops.quantize_activations(x, scale, zp, qmax, want_chansum=False)
                want = torch.clamp(torch.round(x / scale - zp), 0.0, qmax)
                want = torch.nan_to_num(want, nan=0.0).to(torch.uint8)
                assert torch.equal(codes, want.contiguous()), (bits, hex(m), e)


@pytest.mark.parametrize("operand", ["weight", "bias", "quant", "lut"])
def test_layer_pass_refuses_operands_it_cannot_read(dev, operand):
    """Operands go to the library as pointers: another type, another device, another length or stride is an error here,
    before anything is launched."""
    import approx_ops
    x = torch.rand(2, 4, 6, 6, device=dev)
    good = dict(weight=torch.randn(8, 4, 3, 3, device=dev), bias=torch.zeros(8, device=dev),
                quant=torch.tensor([0.01, 0.0, 0.02, -60.0], device=dev), lut=torch.zeros(17408, dtype=torch.uint16, device=dev))
    bad = [good[operand].cpu()]
    if operand != "lut":
        bad += [good[operand].half(), good[operand].double()]
    if operand in ("bias", "quant"):
        t = good[operand]
        bad += [t[:-1], torch.zeros(2 * t.numel(), device=dev)[::2], t[:1].expand(t.numel())]
    launches = approx_ops.library().lutgemm_kernel_launches()

    def layer_pass(kw):
        return approx_ops.conv2d_layer_pass(x, kw["weight"], kw["bias"], kw["quant"], 127.0, 127.0, kw["lut"], 1, 1, 1)

    for b in bad:
        with pytest.raises(RuntimeError):
            layer_pass({**good, operand: b})
        if operand in ("weight", "quant"):
            with pytest.raises(RuntimeError):
                approx_ops.layer_weight_prep(b if operand == "weight" else good["weight"],
                                             b if operand == "quant" else good["quant"], 127.0)
    assert approx_ops.library().lutgemm_kernel_launches() == launches
    layer_pass(good)


def test_a_layer_runs_on_slower_kernels_where_the_fast_ones_do_not_fit(dev, monkeypatch):
    """Workspaces beyond 64 kilobytes cannot be had (an allocator that says so): the operator, a convolution and a
    linear layer give the results of the kernels that need less; what no kernel can do without is an error as before."""
    import approx_ops
    import self_ops
    from lutgemm_layers import AppConv2d, AppLinear
    from lutgemm_luts import synthetic_multiplier, window_difference_gradients
    fp = synthetic_multiplier(7, seed=0)
    self_ops.set_lookup_tables(dev, fp, *window_difference_gradients(fp, 8), 7)
    torch.manual_seed(0)
    conv = AppConv2d(64, 128, 3, 1, 1, bias=True, a_bits=7, w_bits=7, conv_impl="layer").to(dev).train()
    lin = AppLinear(300, 700, a_bits=7, w_bits=7, impl="layer").to(dev).train()
    x, y = torch.rand(4, 64, 10, 10, device=dev), torch.randn(350, 300, device=dev)
    a = torch.randint(0, 128, (400, 200), device=dev).float()
    w = torch.randint(0, 128, (200, 600), device=dev).float()

    def run():
        out = []
        for f, args in ((conv, (x,)), (lin, (y,)), (self_ops.approx_gemm_op, (a, w))):
            args = [t.clone().requires_grad_(True) for t in args]
            conv.zero_grad()
            lin.zero_grad()
            r = f(*args)
            r.backward(torch.ones_like(r))
            out += [r.detach()] + [t.grad for t in args] + [p.grad.clone() for m in (conv, lin) for p in m.parameters() if p.grad is not None]
        return out

    want = run()
    empty, refused = torch.empty, []

    def short(*size, **kw):
        n = size[0] if isinstance(size[0], int) else 0
        if kw.get("dtype") == torch.uint8 and len(size) == 1 and n > 1 << 16:
            refused.append(n)
            raise torch.OutOfMemoryError("no room")
        return empty(*size, **kw)
    monkeypatch.setattr(torch, "empty", short)
    got = run()
    assert len(refused) >= 6
    for g, r in zip(got, want):
        assert torch.linalg.vector_norm(g - r) <= 1e-5 * torch.linalg.vector_norm(r)
    # 4096 rows: the weight gradient needs its code copy under either choice
    a = torch.randint(0, 128, (4096, 200), device=dev).float().requires_grad_(True)
    r = self_ops.approx_gemm_op(a, w.requires_grad_(True))
    with pytest.raises(torch.OutOfMemoryError):
        r.sum().backward()


@pytest.mark.parametrize("cout,batch,held", [(16, 64, False), (31, 64, False), (16, 48, True), (32, 64, True), (64, 64, True)])
def test_narrow_layers_hold_no_large_code_copy_for_the_backward_pass(dev, cout, batch, held):
    import self_ops
    from lutgemm_layers import AppConv2d, AppLinear
    from lutgemm_luts import synthetic_multiplier, window_difference_gradients
    self_ops.set_lookup_tables(dev, synthetic_multiplier(7, seed=0), *window_difference_gradients(synthetic_multiplier(7, seed=0), 8), 7)
    conv = AppConv2d(16, cout, 3, 1, 1, bias=False, a_bits=7, w_bits=7, conv_impl="layer").to(dev).train()
    lin = AppLinear(144, cout, a_bits=7, w_bits=7, impl="layer").to(dev).train()
    for out in (conv(torch.rand(batch, 16, 32, 32, device=dev)), lin(torch.rand(batch * 1024, 144, device=dev))):
        fn = out.grad_fn
        while not hasattr(fn, "codes_t"):
            fn = fn.next_functions[0][0]
        assert (fn.codes_t is not None) == held
        out.sum().backward()


@pytest.mark.parametrize("B,Cin,H,W,Cout,kh,kw,st,p,d", GEOMS + [(4, 40, 17, 19, 70, 3, 3, 1, 2, 2), (2, 16, 30, 30, 24, 3, 3, 2, 3, 3)])
@pytest.mark.parametrize("channels_last", [False, True])
def test_layer_pass_equals_its_steps(dev, B, Cin, H, W, Cout, kh, kw, st, p, d, channels_last):
    """The one-call forward pass of a convolution layer against the five calls it stands for: identical outputs."""
    import approx_ops
    from lutgemm_luts import synthetic_multiplier
    from oracle import oracle_np as O
    torch.manual_seed(Cout)
    fmt = torch.channels_last if channels_last else torch.contiguous_format
    x = torch.rand(B, Cin, H, W, device=dev).contiguous(memory_format=fmt)
    weight = torch.randn(Cout, Cin, kh, kw, device=dev).contiguous(memory_format=fmt)
    bias = torch.randn(Cout, device=dev)
    quant = torch.tensor([1 / 127, 0.0, 0.05, -63.0], device=dev)
    s_a, z_a, s_w, z_w = (quant[i:i + 1] for i in range(4))
    lut = torch.from_numpy(O.pack_padded(synthetic_multiplier(7, seed=1), 7, np.uint16)).to(dev)
    out, codes, wmat, codes_t = approx_ops.conv2d_layer_pass(x, weight, bias, quant, 127.0, 127.0, lut, st, p, d)
    codes_, chansum = approx_ops.quantize_activations(x, s_a, z_a, 127.0)
    wmat_, wsum = approx_ops.layer_weight_prep(weight, quant, 127.0)
    sumw_t, taps = approx_ops.layer_cross_terms(wsum, Cin, H, W, kh, kw, st, p, d)
    box = approx_ops.layer_window_sum(chansum, kh, kw, st, p, d)
    out_, codes_t_ = approx_ops.approx_conv2d_forward_layer(codes_, wmat_, lut, kh, kw, st, p, d, box, sumw_t, taps, s_a, s_w, z_a,
                                                            z_w, bias)
    assert torch.equal(codes, codes_) and torch.equal(wmat, wmat_) and torch.equal(out, out_)
    assert (codes_t is None) == (codes_t_ is None) and (codes_t is None or torch.equal(codes_t, codes_t_))


def test_ranges_of_tensors_in_any_memory_order(dev):
    """A layer's fused range update on inputs that are contiguous, channels-last, permuted otherwise, sliced or expanded."""
    from lutgemm_layers import AppConv2d, _in_memory_order
    base = torch.randn(4, 6, 8, 10, device=dev)
    wide = torch.randn(4, 6, 8, 20, device=dev)
    for x in (base, base.contiguous(memory_format=torch.channels_last), base.permute(0, 1, 3, 2), base.permute(1, 0, 2, 3),
              wide[..., ::2], wide[:, :, :, 3:13], base[:, :1].expand(-1, 6, -1, -1), base.reshape(4, 6, 80)):
        y = _in_memory_order(x)
        assert y.numel() == x.numel() and torch.equal(torch.stack(torch.aminmax(y)), torch.stack((x.min(), x.max())))
        if x.dim() == 4:
            ref, new = (AppConv2d(x.shape[1], 3, 3, a_bits=7, w_bits=7, conv_impl=impl).to(dev).train() for impl in ("fused", "layer"))
            new.load_state_dict(ref.state_dict())
            ref._refresh(x, ref.weight)
            new._refresh(x, new.weight, fused=True)
            assert torch.equal(ref.quant, new.quant)
