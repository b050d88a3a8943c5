"""GPU tests of the gradient kernels on 16-bit slabs where most table entries in use are zero or small against the table's extremes:
dead channels, sparse activations, a table with a few outliers.  A sum over entries that are all zero is exactly zero.

Tolerance: as for the other gradient kernels, 1e-5 of the sum of the absolute terms.  Entries are exact fp32 numbers whatever else
the table holds, so the bound of fewer than 100 additions in a chain, 6e-6, holds for these sums too."""
import numpy as np
import pytest
import torch

from oracle import oracle_np as O
from test_gpu_packed_slab import backward, check, problem

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.fail("gpu-marked test started without a CUDA device")
    import approx_ops
    approx_ops.library()
    return torch.device("cuda:0")


@pytest.fixture(params=["rows", "wide", "tall"])
def tile(request):
    import approx_ops
    approx_ops.set_kernel_choice(backward="slab", grad_tile=request.param)
    yield request.param
    approx_ops.set_kernel_choice()


def tables(bits, least, most, small=None):
    """Entries from `least` to `most`, zero where either code is zero; with `small` all but one of each extreme within +-small."""
    rng = np.random.default_rng(bits)
    q = 1 << bits
    out = []
    for _ in range(2):
        t = rng.integers(-small, small + 1, (q, q)) if small else rng.integers(least, most + 1, (q, q))
        t[q - 1, q - 2], t[q - 1, q - 1] = least, most
        t[0, :] = t[:, 0] = 0
        out.append(O.pack_padded(t, bits, np.int16))
    return out


@pytest.mark.parametrize("bits", [4, 6, 7, 8])
@pytest.mark.parametrize("share", [0.5, 0.9, 0.99])
@pytest.mark.parametrize("M,K,N", [(1100, 20, 200), (200, 20, 1100)])
def test_codes_of_which_most_are_zero(dev, oracle_c, tile, bits, share, M, K, N):
    la, lw = tables(bits, -500, 2040)
    a, w, gc = problem(bits, M, K, N, 7)
    rng = np.random.default_rng(8)
    a[rng.random(a.shape) < share] = 0
    w[rng.random(w.shape) < share] = 0
    a[:, 3] = 0  # a dead channel
    w[5] = 0
    ga, gw = backward(dev, gc, a, w, la, lw)
    # (a = 0 makes every entry of both tables zero, and so does w = 0)
    assert (gw[3] == 0).all() and (ga[:, 3] == 0).all() and (gw[5] == 0).all() and (ga[:, 5] == 0).all()
    r_ga, r_gw, r_gaa, r_gwa = oracle_c.backward_f64(gc, a, w, la, lw, bits)
    check(ga, r_ga, r_gaa)
    check(gw, r_gw, r_gwa)


@pytest.mark.parametrize("bits", [4, 6, 7, 8])
@pytest.mark.parametrize("least,most,small", [(-2000, 8000, 60), (-8191, 32767, 10), (-32768, 32767, 10)])
def test_tables_with_outliers(dev, oracle_c, tile, bits, least, most, small):
    la, lw = tables(bits, least, most, small)
    a, w, gc = problem(bits, 1100, 20, 1100, 9)
    a %= (1 << bits) - 1  # the outliers' row stays unused
    ga, gw = backward(dev, gc, a, w, la, lw)
    r_ga, r_gw, r_gaa, r_gwa = oracle_c.backward_f64(gc, a, w, la, lw, bits)
    check(ga, r_ga, r_gaa)
    check(gw, r_gw, r_gwa)
