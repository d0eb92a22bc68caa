"""Linears of 3 to 16 rows whose activations are reordered first (k_interleave_x), at the edges of that rule and of the order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,N,th,M", [
    (5504, 4100, 128, 5),       # the last tile pair is half there
    (4096, 4608, 128, 5),       # just below the rule, plain rows
    (4099, 7500, 128, 4),       # K odd: reordered whatever the size
    (5000, 6016, 128, 7),       # the last tile is not whole
    (4096, 4096, 1024, 9),      # entry points, two sets of rows
    (3000, 10000, 64, 16),      # short tiles, all rows
    (6200, 4096, 2048, 3),      # entry points, the last tile short
])
def test_reordered_activations(K, N, th, M):
    import comp_inference_b200 as ci
    g = torch.Generator("cuda").manual_seed(K + M)
    W = (torch.randn(K, N, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    c = ci.compress_weight_cuda(W, th, 32)
    m = ci.RansLinear(K, N, c["tile_height"], 32).load_compressed(c).prepare()
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    y = m(x).double()
    ref = x.double() @ W.double()
    # bf16 result: half a unit in the last place, 2^-9; K products summed in 32 bits, truncating: K x 2^-23 of their magnitudes
    bound = ref.abs() * 2.0 ** -8 + (x.double().abs() @ W.double().abs()) * (K * 2.0 ** -23)
    assert bool(((y - ref).abs() <= bound).all())
