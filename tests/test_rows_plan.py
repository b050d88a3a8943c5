"""How the gradient kernel with one thread per output row deals out its work, and where it is chosen, without a GPU."""
import os
import subprocess

import pytest

import host_dispatch as H


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return H.Library(H.build(tmp_path_factory.mktemp("host")))


def test_plan_covers_its_work(tmp_path):
    exe = str(tmp_path / "plan")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", exe, os.path.join(H.HERE, "rows_plan_check.cpp"), "-I",
                    os.path.join(H.ROOT, "appmult-aware-retraining_b200", "csrc"), "-I", os.path.join(H.ROOT, "include"), "-I",
                    os.path.join(cuda, "include")], check=True)
    res = subprocess.run([exe], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout


ROWS, PACKED, BCAST = "slab_grad_rows_kernel", "slab_grad_packed_kernel", "ga_colbcast_kernel"


@pytest.mark.parametrize("bits,B,Cin,Cout,h,k,stride,kernel,without", [
    (7, 256, 64, 64, 32, 3, 1, ROWS, ROWS), (8, 64, 256, 64, 56, 1, 1, ROWS, ROWS), (8, 256, 256, 512, 8, 3, 2, ROWS, None),
    (7, 1, 64, 64, 8, 3, 1, PACKED, PACKED), (7, 64, 256, 256, 56, 3, 1, ROWS, PACKED), (8, 16, 128, 256, 10, 3, 1, ROWS, BCAST),
    (7, 2, 256, 1024, 6, 3, 1, PACKED, None)])
def test_image_gradients(lib, bits, B, Cin, Cout, h, k, stride, kernel, without):
    """One thread per pixel where the caller brings its workspace; without one the kernels that need none, or a refusal where a
    buffer has always been asked for (`without` None)."""
    p = lib.p
    conv = (bits, B, Cin, h, h, Cout, k, k, stride, k // 2, 1)
    need = lib.query("lutgemm_conv2d_backward_ws_scratch_bytes", *conv, H.CODES_GIVEN)
    for nbytes, expected in ((1 << 40, kernel), (need, kernel), (0, without if need else kernel)):
        rc, calls = lib.call("lutgemm_conv2d_backward_ws", p, p, p, p, None, p, p, *conv, None, p if nbytes else None, H.Size(nbytes), None)
        assert rc == (H.OK if expected else H.E_SCRATCH)
        assert {c[0] for c in calls} & {ROWS, PACKED, BCAST} == ({expected} if expected else set())


def test_operator_gradients_fall_back_where_the_buffer_is_small(lib):
    p, shape = lib.p, (7, 4096, 512, 4096)
    need, least = (lib.query("lutgemm_backward_ws_scratch_bytes", *shape, f) for f in (0, H.LEAST))
    assert least <= need
    for nbytes, kernel in ((need, "slab_grad_rows_kernel"), (least, "slab_grad_rows_kernel" if least == need else "slab_grad_tall_kernel")):
        rc, calls = lib.call("lutgemm_backward", p, p, p, p, p, p, p, *shape, p, H.Size(nbytes), None)
        assert rc == H.OK and kernel in {c[0] for c in calls}
