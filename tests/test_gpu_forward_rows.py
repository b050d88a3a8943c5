"""GPU tests of the forward kernel with two output rows per thread (1024 rows x 32 columns) at the sizes where it can go wrong:
odd K, remainders of its tiles, units and operand stages, tiles cut across CTAs and whole tiles of which a CTA takes several,
weight rows that are not 16-byte aligned, and the layer's de-quantisation on the way out.  Sums are whole numbers, so they
equal the broadcast kernel's; so do layer outputs, whose roundings are in the same order."""
import numpy as np
import pytest
import torch

from oracle import oracle_np as O
from test_gpu_packed_slab import problem

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.fail("gpu-marked test started without a CUDA device")
    import approx_ops
    approx_ops.library()
    return torch.device("cuda:0")


def run(dev, family, bits, a, w, lut, layer):
    import approx_ops
    (M, K), N = a.shape, w.shape[1]
    box, sumw, taps = a.sum(dim=1, dtype=torch.float32), w.sum(dim=0, dtype=torch.float32).view(1, N), torch.full((1,), float(K), device=dev)
    q = [torch.tensor([v], device=dev) for v in (0.013, 0.021, -3.0, -61.0)]
    try:
        approx_ops.set_kernel_choice(forward=family)
        if layer:
            out, _ = approx_ops.approx_gemm_forward_layer(a, w, lut, box, sumw, taps, *q, torch.arange(N, device=dev, dtype=torch.float32))
        else:
            c = torch.full((M, N), 7, dtype=torch.int32, device=dev)
            approx_ops.approx_gemm_forward(a, w, c.view(torch.uint32), lut)
            out = c
        torch.cuda.synchronize()
        assert approx_ops.device_error() == 0
        return out
    finally:
        approx_ops.set_kernel_choice()


@pytest.mark.parametrize("layer", [False, True])
@pytest.mark.parametrize("bits", [4, 6, 7, 8])
@pytest.mark.parametrize("M,K,N", [(1024, 1, 32), (1023, 2, 31), (1025, 3, 33), (1, 4, 1), (2050, 5, 64), (3000, 17, 100), (700, 63, 48), (40, 301, 70),
                                   (1024 * 150, 21, 32), (1024 * 297 - 100, 70, 20), (5000, 777, 333)])
def test_sums_and_layer_outputs(dev, bits, M, K, N, layer):
    a, w, _ = problem(bits, M, K, N, bits + M)
    # (entries over all 16 bits; with a layer below 2^12, so that the sums are exact in fp32 whatever way they are added)
    lut = O.pack_padded(np.random.default_rng(bits).integers(0, 2 ** 12 if layer else 2 ** 16, (1 << bits, 1 << bits)), bits, np.uint16)
    a, w, lut = (torch.from_numpy(v).to(dev) for v in (a, w, lut))
    assert torch.equal(run(dev, "rows", bits, a, w, lut, layer), run(dev, "rowbcast", bits, a, w, lut, layer))
