"""Which decoder restores a weight whose tiles are deep: exact, and not by the generic kernel where a staged one has room.

Incompressible exponents make a tile's byte block half its height in rows, so a window of 128-byte rows (decode4.cu) stops fitting
at 1500 rows or so and one of 64-byte rows (decode2.cu) at 3000."""
import pytest
import torch

from conftest import captured_kernels

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
    from comp_inference_b200 import _lib
    g = torch.Generator("cuda").manual_seed(th + exps + N)
    bits = torch.randint(0, exps, (th, N), generator=g, device="cuda") << 7 | torch.randint(0, 128, (th, N), generator=g, device="cuda")
    W = bits.to(torch.int16)
    c = ci.compress_weight_cuda(W.view(torch.bfloat16), th, 32)
    assert c["tile_height"] == th
    w, keep = _lib.tiled_weight(c["rans_exp_stream"], c["rans_exp_states"], c["rans_exp_tables"], c["rans_exp_slot_map"],
                                c["rans_exp_tile_offsets"], c["rans_exp_tile_max_lens"], c["rans_man_raw"], th, N, th, 32,
                                want_max=True)
    out = torch.zeros_like(W)

    def call():
        _lib.check(_lib.load().ci_decode_bf16(w, out.data_ptr(), torch.cuda.current_stream().cuda_stream))
    call()
    assert torch.equal(out, W)
    launched = captured_kernels(call)
    assert staged == ("k_decode2" in launched or "k_decode4" in launched) and ("k_decode_tiled" in launched) == (not staged)


@pytest.mark.parametrize("K,N,th,kernel", [
    (4096, 4096, 128, "k_decode4"),
    (4096, 22016, 128, "k_decode4"),
    (2048, 2048, 128, "k_decode2"),     # one warp a scheduler: two streams a lane start sooner
    (777, 1001, 128, "k_decode2"),
    (4096, 11008, 1024, "k_decode2"),   # long streams, few tiles
])
def test_choice_of_decoder(K, N, th, kernel):
    import comp_inference_b200 as ci
    from comp_inference_b200 import _lib
    W = (torch.randn(K, N, generator=torch.Generator("cuda").manual_seed(K), device="cuda") * 0.02).to(torch.bfloat16)
    c = ci.compress_weight_cuda(W, th, 32)
    w, keep = _lib.tiled_weight(c["rans_exp_stream"], c["rans_exp_states"], c["rans_exp_tables"], c["rans_exp_slot_map"],
                                c["rans_exp_tile_offsets"], c["rans_exp_tile_max_lens"], c["rans_man_raw"], K, N, th, 32, want_max=True)
    out = torch.empty_like(W)

    def call():
        _lib.check(_lib.load().ci_decode_bf16(w, out.data_ptr(), torch.cuda.current_stream().cuda_stream))
    call()
    assert torch.equal(out.view(torch.int16), W.view(torch.int16))
    assert kernel in captured_kernels(call)
