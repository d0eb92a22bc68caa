"""The linear on a weight stored transposed (linear_t4.cu) where its sums stay in registers and where a CTA works on two groups."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _call(c, shape, x):
    import comp_inference_b200 as ci
    return ci.fused_rans_linear_transposed_triton(
        x, c["rans_exp_stream"], initial_states=c["rans_exp_states"], tables=c["rans_exp_tables"], slot_map=c["rans_exp_slot_map"],
        weight_shape=shape, tile_offsets=c["rans_exp_tile_offsets"], tile_max_lens=c["rans_exp_tile_max_lens"],
        tile_k=c["tile_height"], tile_n=c["tile_width"], mantissas=c["rans_man_raw"])


@pytest.mark.parametrize("V,H,th", [
    (17, 40, 16),          # one chunk of eight rows, columns beyond the matrix
    (40000, 16, 32),       # one column block a group: a CTA has many groups
    (5003, 200, 64),       # two chunks, the last group lacks tiles
    (20000, 130, 128),     # four chunks, odd pairs of columns
    (3001, 333, 96),       # three chunks, activations at odd addresses
    (7000, 1027, 1024),    # entry points
    (2000, 512, 256),      # entry points, one group a CTA or none
])
@pytest.mark.parametrize("M", [1, 2, 3])
def test_transposed_linear(V, H, th, M):
    import comp_inference_b200 as ci
    g = torch.Generator("cuda").manual_seed(V + M)
    W = (torch.randn(V, H, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    c = ci.compress_weight_cuda(W, th, 32)
    x = torch.randn(M, H, generator=g, device="cuda").to(torch.bfloat16)
    for _ in range(2):                                   # the second call finds the tickets as the first one left them
        y = _call(c, (V, H), x).double()
        ref = x.double() @ W.double().t()
        # bf16 result: half a unit in the last place, 2^-9; H products summed in 32 bits, truncating: H x 2^-23 of their magnitudes
        bound = ref.abs() * 2.0 ** -8 + (x.double().abs() @ W.double().abs().t()) * (H * 2.0 ** -23)
        assert bool(((y - ref).abs() <= bound).all())


@pytest.mark.parametrize("M", [1, 2])
def test_infinite_weight_stays_in_its_row(M):
    import comp_inference_b200 as ci
    V, H = 600, 256
    g = torch.Generator("cuda").manual_seed(5)
    W = (torch.randn(V, H, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    W[77, 3], W[300, 200] = float("inf"), float("nan")
    c = ci.compress_weight_cuda(W, 128, 32)
    x = torch.randn(M, H, generator=g, device="cuda").to(torch.bfloat16)
    y = _call(c, (V, H), x)
    bad = (~torch.isfinite(y)).any(0).nonzero().flatten().tolist()
    assert bad == [77, 300]


@pytest.mark.parametrize("V,H,th,M", [
    (600, 250, 128, 1),    # sums in registers, the last column block has ten columns
    (600, 90, 64, 2),
    (600, 333, 16, 8),     # sums in shared memory
    (1500, 1003, 1024, 1), # entry points
    (1500, 1003, 1024, 5),
])
def test_infinite_weight_beside_missing_columns(V, H, th, M):
    import comp_inference_b200 as ci
    g = torch.Generator("cuda").manual_seed(V + H)
    W = (torch.randn(V, H, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    W[7, H // 16 * 16], W[V - 1, H // 16 * 16], W[40, H - 1] = float("inf"), float("-inf"), float("inf")
    c = ci.compress_weight_cuda(W, th, 32)
    x = torch.randn(M, H, generator=g, device="cuda").to(torch.bfloat16)
    y = _call(c, (V, H), x).double()
    ref = x.double() @ W.double().t()
    inf = ref.isinf()
    assert inf.sum() == 3 * M and torch.equal(y[inf], ref[inf])
    Wf = torch.where(W.isinf(), torch.zeros_like(W), W).double()
    bound = ref.abs() * 2.0 ** -8 + (x.double().abs() @ Wf.abs().t()) * (H * 2.0 ** -23)   # as above
    assert bool(((y - ref).abs() <= bound)[~inf].all())
