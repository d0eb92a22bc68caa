"""Edges of the dispatch rules and of the tiles of the kernels, at the sizes where a branch begins or a remainder is
left, against fp32 products of the exactly decoded weight."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _weight(K, N, seed=3):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(K, N, generator=g) * 0.02).to(torch.bfloat16).cuda()


def _close(y, ref, tol=1e-2):
    return float((y.float() - ref).abs().max() / ref.abs().max()) <= tol


# tall tiles: one pair of tile rows, a lone upper tile, a lower tile that ends early, several pairs, windows that fit
# twice / once per warp; many units per multiprocessor with 9..16 rows: activations reordered first
@pytest.mark.parametrize("K,N,th,M", [(1024, 256, 512, 1), (1536, 96, 512, 3), (2056, 64, 1024, 2), (3000, 96, 1024, 16),
                                      (4096, 64, 1024, 9), (768, 2048, 256, 1), (600, 132, 512, 5),
                                      (2048, 8192, 128, 16), (2056, 8196, 128, 11), (4096, 8192, 64, 5)])
@pytest.mark.parametrize("split_k", [0, 8])
def test_linear_dispatch_edges(K, N, th, M, split_k):
    import comp_inference_b200 as ci
    from comp_inference_b200 import _lib
    W = _weight(K, N)
    c = ci.compress_weight_cuda(W, th, 32)
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).cuda()
    bias = torch.randn(N, generator=torch.Generator().manual_seed(N)).to(torch.bfloat16).cuda()
    y = ci.fused_rans_linear_triton(
        x, c["rans_exp_stream"], c["rans_exp_states"], c["rans_exp_tables"], c["rans_exp_slot_map"], (K, N),
        c["rans_exp_tile_offsets"], c["rans_exp_tile_max_lens"], c["tile_height"], c["tile_width"], c["rans_man_raw"],
        bias=bias, SPLIT_K=split_k)
    assert _close(y, x.float() @ W.float() + bias.float())
    assert _lib.kernel_status(x.device) == 0
