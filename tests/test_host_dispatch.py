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
