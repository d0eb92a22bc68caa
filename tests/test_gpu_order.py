"""Linears of 3 to 16 rows whose activations are reordered first (k_interleave_x), at the edges of that rule and of the order."""
import pytest
import torch

from conftest import captured_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,N,th,M,reordered", [
    (5504, 4100, 128, 5, True),     # the last tile pair is half there
    (4096, 4608, 128, 5, False),    # just below the rule, plain rows
    (4099, 7500, 128, 4, True),     # K odd: reordered whatever the size
    (5000, 6016, 128, 7, True),     # the last tile is not whole
    (4096, 4096, 1024, 9, False),   # entry points, two sets of rows, just below the rule
    (4096, 4096, 1024, 16, True),   # the same above it
    (4096, 7168, 1024, 5, True),    # entry points, one set of rows
    (3000, 10000, 64, 16, True),    # short tiles, all rows
    (6200, 4096, 2048, 3, False),   # entry points, the last tile short, below the rule
    (6200, 4096, 2048, 9, True),    # the same above it
    (6201, 4096, 2048, 3, True),    # and where K is odd
])
def test_reordered_activations(K, N, th, M, reordered):
    import comp_inference_b200 as ci
    g = torch.Generator("cuda").manual_seed(K + M)
    W = (torch.randn(K, N, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    c = ci.compress_weight_cuda(W, th, 32)
    m = ci.RansLinear(K, N, c["tile_height"], 32).load_compressed(c).prepare()
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    y = m(x).double()
    launched = captured_kernels(lambda: m(x))
    assert "k_linear_mma4" in launched and ("k_interleave_x" in launched) == reordered
    ref = x.double() @ W.double()
    # bf16 result: half a unit in the last place, 2^-9; K products summed in 32 bits, truncating: K x 2^-23 of their magnitudes
    bound = ref.abs() * 2.0 ** -8 + (x.double().abs() @ W.double().abs()) * (K * 2.0 ** -23)
    assert bool(((y - ref).abs() <= bound).all())
