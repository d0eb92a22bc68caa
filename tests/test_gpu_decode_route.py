"""Which decoder restores a weight whose tiles are deep: exact, and not by the generic kernel where a staged one has room.

Incompressible exponents make a tile's byte block half its height in rows, so a window of 128-byte rows (decode4.cu) stops fitting
at 1500 rows or so and one of 64-byte rows (decode2.cu) at 3000."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("th,exps,staged", [
    (4096, 32, True),      # 5 bits a symbol, 1280 rows: both have room
    (4096, 64, True),      # 1540 rows: above the limit of 128-byte rows
    (4096, 256, True),     # 2050 rows
    (5632, 256, True),     # 2820 rows: just below the limit of 64-byte rows
    (8192, 256, False),    # 4100 rows: neither
])
@pytest.mark.parametrize("N", [64, 2000])
def test_deep_tiles(th, exps, staged, N):
    import comp_inference_b200 as ci
    from torch.profiler import ProfilerActivity, profile
    g = torch.Generator("cuda").manual_seed(th + exps + N)
    bits = torch.randint(0, exps, (th, N), generator=g, device="cuda") << 7 | torch.randint(0, 128, (th, N), generator=g, device="cuda")
    W = bits.to(torch.int16).view(torch.bfloat16)
    c = ci.compress_weight_cuda(W, th, 32)
    assert c["tile_height"] == th
    args = dict(initial_states=c["rans_exp_states"], tables=c["rans_exp_tables"], slot_map=c["rans_exp_slot_map"], weight_shape=(th, N),
                tile_offsets=c["rans_exp_tile_offsets"], tile_max_lens=c["rans_exp_tile_max_lens"], tile_k=th, tile_n=32,
                mantissas=c["rans_man_raw"])
    call = lambda: ci.rans_decompress_bf16(c["rans_exp_stream"], **args)
    assert torch.equal(call().view(torch.int16), W.view(torch.int16))
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    kernels = [e.key for e in p.key_averages() if "k_decode" in e.key]
    assert len(kernels) == 1
    assert staged == any(k in kernels[0] for k in ("k_decode2", "k_decode4")), kernels
