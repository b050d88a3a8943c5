"""A backward call with a scratch buffer of exactly the size that the library asks for runs, and runs the kernels that a buffer without
limit would: sizes drawn over the range that the entry points take, odd ones among them, without a GPU."""
import math
import random

import pytest

import host_dispatch as H


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return H.Library(H.build(tmp_path_factory.mktemp("host")))


def log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def conv(rng):
    k = rng.choice([1, 2, 3, 3, 5, 7])
    h, w = (log_uniform(rng, max(k, 4), 64) for _ in "hw")
    return (rng.choice([4, 6, 7, 8]), log_uniform(rng, 1, 256), log_uniform(rng, 3, 512), h, w, log_uniform(rng, 2, 1024), k, k,
            rng.choice([1, 1, 2, 3]), rng.choice([0, k // 2]), 1)


def convolutions():
    rng = random.Random(1)
    # (the first four were refused, or ran on slower kernels, with the size that the query named)
    return [(7, 98, 61, 41, 41, 950, 3, 3, 1, 1, 1), (7, 127, 24, 46, 46, 582, 5, 5, 1, 2, 1), (7, 10, 45, 54, 54, 75, 3, 3, 1, 1, 1),
            (7, 126, 30, 16, 47, 982, 3, 3, 1, 0, 1)] + [conv(rng) for _ in range(2000)]


@pytest.mark.parametrize("gx,gw", [(True, True), (True, False), (False, True)])
def test_convolution_backward(lib, gx, gw):
    p, big = lib.p, H.Size(1 << 40)
    for shape in convolutions():
        args = (p, p, p, p if gx else None, p if gw else None, p, p, *shape)
        need = lib.query("lutgemm_conv2d_backward_scratch_bytes", *shape)
        exact = lib.call("lutgemm_conv2d_backward", *args, p, H.Size(need), None)
        assert exact[0] == H.OK and exact == lib.call("lutgemm_conv2d_backward", *args, p, big, None), shape
        for codes, flag in ((None, 0), (p, H.CODES_GIVEN)):
            need = lib.query("lutgemm_conv2d_backward_ws_scratch_bytes", *shape, flag)
            exact = lib.call("lutgemm_conv2d_backward_ws", *args, codes, p, H.Size(need), None)
            assert exact[0] == H.OK and exact == lib.call("lutgemm_conv2d_backward_ws", *args, codes, p, big, None), shape
            least = lib.query("lutgemm_conv2d_backward_ws_scratch_bytes", *shape, flag | H.LEAST)
            assert lib.call("lutgemm_conv2d_backward_ws", *args, codes, p, H.Size(least), None)[0] == H.OK, shape


def products():
    rng = random.Random(2)
    # (the first six: the activation gradient alone ran on a slower kernel with the size that the query named)
    return [(6, 5104, 1095, 2537), (6, 3631, 3095, 670), (4, 3195, 2987, 1832), (8, 1673, 2932, 667), (6, 4776, 3739, 1468),
            (4, 1396, 2477, 3692)] + [
        (rng.choice([4, 6, 7, 8]), log_uniform(rng, 1, 16384), log_uniform(rng, 1, 8192), log_uniform(rng, 1, 8192)) for _ in range(4000)]


@pytest.mark.parametrize("ga,gw", [(True, True), (True, False), (False, True)])
def test_operator_backward(lib, ga, gw):
    p, big = lib.p, H.Size(1 << 40)
    for shape in products():
        args = (p, p, p, p if ga else None, p if gw else None, p, p, *shape)
        need = lib.query("lutgemm_backward_scratch_bytes", *shape)
        exact = lib.call("lutgemm_backward", *args, p, H.Size(need), None)
        assert exact[0] == H.OK and exact == lib.call("lutgemm_backward", *args, p, big, None), shape
        for codes, flag in ((None, 0), (p, H.CODES_GIVEN)):
            need, least = (lib.query("lutgemm_backward_ws_scratch_bytes", *shape, flag | f) for f in (0, H.LEAST))
            exact = lib.call("lutgemm_backward_ws", *args, codes, p, H.Size(need), None)
            assert exact[0] == H.OK and exact == lib.call("lutgemm_backward_ws", *args, codes, p, big, None), shape
            assert lib.call("lutgemm_backward_ws", *args, codes, p, H.Size(least), None)[0] == H.OK, shape
