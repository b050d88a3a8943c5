"""Host code of the library without a GPU: sizes it asks for, calls it refuses and kernels it chooses."""
import os
import subprocess
import sys

import pytest

import host_dispatch as H

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return H.Library(H.build(tmp_path_factory.mktemp("host")))


@pytest.mark.parametrize("k,stride", [(11, 1), (12, 1), (23, 1), (50, 1), (50, 2)])
def test_scratch_query_for_windows_of_many_taps(lib, k, stride):
    """An image gradient has room for 128 taps per stride class and is refused beyond; the query for its scratch buffer,
    in a process of its own, must neither fail nor ask for more than the weight gradient needs."""
    code = ("import sys; sys.path[:0] = %r; import host_dispatch as H; L = H.Library(%r); "
            "print(L.query('lutgemm_conv2d_backward_scratch_bytes', 7, 2, 8, 64, 64, 64, %d, %d, %d, 0, 1))"
            % (sys.path[:4] + [HERE], lib.lib._name, k, k, stride))
    res = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    need, p = H.Size(int(res.stdout)), lib.p
    conv = (7, 2, 8, 64, 64, 64, k, k, stride, 0, 1)
    assert lib.call("lutgemm_conv2d_backward", p, p, p, None, p, p, p, *conv, p, need, None)[0] == H.OK
    rc, _ = lib.call("lutgemm_conv2d_backward", p, p, p, p, None, p, p, *conv, p, need, None)
    assert rc == (H.OK if k * k <= 128 else H.E_TOOLARGE)


@pytest.mark.parametrize("K", [2097120, 2097121, 2200001, 4194240, 4194256, 9000001])
def test_long_k_is_not_refused(lib, K):
    """Few rows and a long K: the slab kernels' transposed code copy is made in as many launches as its grid needs."""
    p, big = lib.p, H.Size(1 << 40)
    rc, calls = lib.call("lutgemm_forward_ws", p, p, p, p, 4, 16, K, 64, p, big, None)
    assert rc == H.OK and calls[-1][0] == "slab_fwd_kernel"
    per_launch = 65535 * (64 if K % 16 == 0 else 32)
    assert sum(name.startswith("transpose") for name, _ in calls) == (K + per_launch - 1) // per_launch
    assert lib.call("lutgemm_backward", p, p, p, p, p, p, p, 4, 16, K, 64, p, big, None)[0] == H.OK


def layer_pass(lib, bits=7, B=4, C=64, h=8, Cout=64, k=3, a_qmax=127.0, scratch_bytes=1 << 40, **null):
    p = lib.p
    ptr = {name: null.get(name, p) for name in ("x", "weight", "quant", "lut", "codes", "wmat", "out", "work", "scratch")}
    s = [H.Size(1)] * 4
    return lib.call("lutgemm_conv2d_layer_pass", ptr["x"], *s, ptr["weight"], *s, None, ptr["quant"], a_qmax, 127.0, ptr["lut"], bits,
                    B, C, h, h, Cout, k, k, 1, 1, 1, ptr["codes"], ptr["wmat"], ptr["out"], ptr["work"], ptr["scratch"],
                    H.Size(scratch_bytes), None)


@pytest.mark.parametrize("bad,status", [
    (dict(bits=5), H.E_BITS), (dict(x=None), H.E_BADARG), (dict(weight=None), H.E_BADARG), (dict(quant=None), H.E_BADARG),
    (dict(lut=None), H.E_BADARG), (dict(codes=None), H.E_BADARG), (dict(wmat=None), H.E_BADARG), (dict(out=None), H.E_BADARG),
    (dict(work=None), H.E_BADARG), (dict(lut=(1 << 40) + 1), H.E_BADARG), (dict(out=(1 << 40) + 2), H.E_BADARG),
    (dict(scratch=(1 << 40) + 8), H.E_BADARG), (dict(a_qmax=256.0), H.E_BADARG), (dict(a_qmax=0.0), H.E_BADARG),
    (dict(k=65, h=80), H.E_BADARG), (dict(B=70000, h=3), H.E_TOOLARGE),
    (dict(B=64, scratch_bytes=64), H.E_SCRATCH),                  # whole tiles, transposed copy only
    (dict(B=8, C=512, scratch_bytes=64), H.E_SCRATCH), (dict(B=8, C=512, scratch=None, scratch_bytes=0), H.E_SCRATCH)])  # cut K
def test_layer_pass_refuses_before_it_launches(lib, bad, status):
    bad = {k: H.ctypes.c_void_p(v) if k in ("lut", "out", "scratch") and v else v for k, v in bad.items()}
    assert layer_pass(lib, **bad) == (status, [])


def test_layer_pass_with_a_small_workspace_where_only_the_estimate_picks_the_slab_kernel(lib):
    assert layer_pass(lib)[1][-1][0] == "conv_epilogue_kernel"  # (K cut, sums in the workspace)
    for kw in (dict(scratch_bytes=64), dict(scratch=None, scratch_bytes=0)):
        rc, calls = layer_pass(lib, **kw)
        assert rc == H.OK and "rowbcast" in calls[-1][0]


@pytest.mark.parametrize("lut,scratch", [((1 << 40) + 1, 1 << 40), (1 << 40, (1 << 40) + 4)])
@pytest.mark.parametrize("scratch_bytes", [64, 1 << 40])
def test_layer_forward_refuses_misaligned_buffers_whatever_the_workspace(lib, lut, scratch, scratch_bytes):
    p = lib.p
    assert lib.call("lutgemm_forward_layer", p, p, H.ctypes.c_void_p(lut), 7, 256, 576, 64, p, p, p, p, p, p, p, None, p,
                    H.ctypes.c_void_p(scratch), H.Size(scratch_bytes), None) == (H.E_BADARG, [])


def test_weight_gradient_without_allocation_follows_a_forced_kernel_family(lib):
    """What fits the fixed array is the need of the kernels that run: 28 MB of codes and 4 blocks of sums for the slab
    kernels, nothing or a few splits for the broadcast kernel."""
    p, shape = lib.p, (4096, 7000, 320)
    try:
        for family, status in ((0, H.E_TOOLARGE), (1, H.OK), (2, H.E_TOOLARGE)):
            lib.lib.lutgemm_set_kernel_choice(0, family, 0)
            rc, calls = lib.call("lutgemm_backward_gw_noalloc", p, p, p, p, p, 8, *shape, None)
            assert rc == status and (rc != H.OK or calls[0][0] == "gw_rowbcast_kernel")
    finally:
        lib.lib.lutgemm_set_kernel_choice(0, 0, 0)


@pytest.mark.parametrize("bits,B,Cin,Cout,h,k,stride", [(7, 64, 256, 256, 56, 3, 1), (6, 256, 64, 64, 32, 3, 1), (8, 256, 256, 512, 8, 3, 2),
                                                        (7, 2, 24, 40, 9, 3, 1), (8, 64, 256, 64, 56, 1, 1)])
def test_backward_scratch_has_no_room_for_codes_that_are_given(lib, bits, B, Cin, Cout, h, k, stride):
    p, pad, ho = lib.p, k // 2, (h + 2 * (k // 2) - k) // stride + 1
    M, K = B * ho * ho, Cin * k * k
    conv = (bits, B, Cin, h, h, Cout, k, k, stride, pad, 1)
    gemm = (bits, M, K, Cout)
    for name, shape in (("lutgemm_conv2d_backward", conv), ("lutgemm_backward", gemm)):
        full, given = (lib.query(name + "_ws_scratch_bytes", *shape, flags) for flags in (0, H.CODES_GIVEN))
        assert full == lib.query(name + "_scratch_bytes", *shape)
        assert full >= K * ((M + 15) // 16 * 16) > 0 and given <= full
        rc, calls = lib.call(name + "_ws", p, p, p, p, p, p, p, *shape, p, p, H.Size(given), None)
        assert rc == H.OK and not any("transpose" in c[0] for c in calls)
        rc_full, calls_full = lib.call(name + "_ws", p, p, p, p, p, p, p, *shape, None, p, H.Size(full), None)
        assert rc_full == H.OK and [c for c in calls_full if "transpose" not in c[0]] == calls
    # one gradient alone: the copy is all that the two needs differ by
    gw_full, gw_given = (lib.query("lutgemm_backward_ws_scratch_bytes", bits, M, K, Cout, f) for f in (0, H.CODES_GIVEN))
    assert gw_full - gw_given <= K * ((M + 15) // 16 * 16) + 15


def test_plan_of_the_packed_gradient_kernels_covers_its_work(tmp_path):
    exe = str(tmp_path / "plan")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", exe, os.path.join(HERE, "packed_plan_check.cpp"), "-I",
                    os.path.join(H.ROOT, "appmult-aware-retraining_b200", "csrc"), "-I", os.path.join(H.ROOT, "include"), "-I",
                    os.path.join(cuda, "include")], check=True)
    res = subprocess.run([exe], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout


@pytest.mark.parametrize("bits,B,C,h", [(7, 64, 256, 56), (7, 256, 256, 56), (7, 64, 512, 28), (6, 256, 64, 32), (4, 1024, 64, 32)])
def test_image_gradient_needs_no_partial_sums_and_weight_gradient_one_block_per_1024_rows(lib, bits, B, C, h):
    """3x3 layers of C channels whose pixel tiles fill the GPU."""
    need = lib.query("lutgemm_conv2d_backward_ws_scratch_bytes", bits, B, C, h, h, C, 3, 3, 1, 1, 1, H.CODES_GIVEN)
    assert need <= (B * h * h + 1023) // 1024 * 9 * C * C * 4


@pytest.mark.parametrize("given", [0, H.CODES_GIVEN])
@pytest.mark.parametrize("bits,B,Cin,Cout,h,k,stride", [(7, 64, 256, 256, 28, 3, 1), (6, 256, 64, 64, 32, 3, 1), (8, 256, 256, 512, 8, 3, 2),
                                                        (7, 1, 64, 256, 8, 3, 1), (8, 64, 256, 64, 56, 1, 1), (7, 8, 64, 1024, 28, 1, 1)])
def test_least_scratch_is_accepted_and_nothing_below_it(lib, given, bits, B, Cin, Cout, h, k, stride):
    p, pad, ho = lib.p, k // 2, (h + 2 * (k // 2) - k) // stride + 1
    codes = p if given else None
    for name, shape in (("lutgemm_conv2d_backward", (bits, B, Cin, h, h, Cout, k, k, stride, pad, 1)),
                        ("lutgemm_backward", (bits, B * ho * ho, Cin * k * k, Cout))):
        need, least = (lib.query(name + "_ws_scratch_bytes", *shape, f | given) for f in (0, H.LEAST))
        assert least <= need

        def status(nbytes):
            return lib.call(name + "_ws", p, p, p, p, p, p, p, *shape, codes, p, H.Size(nbytes), None)[0]
        assert status(least) == H.OK and (least == 0 or status(least - 1) == H.E_SCRATCH)


@pytest.mark.parametrize("bits,B,Cin,Cout,h,k,stride,slab", [
    (7, 256, 64, 64, 32, 3, 1, False), (7, 256, 128, 128, 16, 3, 1, True), (7, 256, 64, 128, 32, 3, 2, False),
    (7, 256, 128, 256, 16, 3, 2, False), (7, 256, 256, 512, 8, 3, 2, True), (8, 256, 64, 64, 32, 3, 1, False),
    (8, 256, 128, 256, 16, 3, 2, False), (8, 256, 256, 512, 8, 3, 2, True), (7, 16, 32, 64, 20, 5, 3, False), (7, 2, 48, 96, 30, 7, 5, False)])
def test_kernel_family_of_image_gradients(lib, bits, B, Cin, Cout, h, k, stride, slab):
    """The choice counts what the busiest SM gets from the tiles of all stride classes (1, 4, 9 and 25 of them here)."""
    p = lib.p
    rc, calls = lib.call("lutgemm_conv2d_backward", p, p, p, p, None, p, p, bits, B, Cin, h, h, Cout, k, k, stride, k // 2, 1, p,
                         H.Size(1 << 40), None)
    names = {c[0] for c in calls}
    assert rc == H.OK and ("slab_grad_packed_kernel" in names, "ga_colbcast_kernel" in names) == (slab, not slab)
