"""The row gather where ids share streams (embedding_group.cu): exact, whatever the ids and however they are spread."""
import math

import pytest
import torch

from conftest import captured_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,H,th", [
    (4000, 512, 64),       # 32 rows a bin
    (4001, 1100, 128),     # 63 bins of 65 ids: too few, ungrouped
    (5001, 1100, 128),     # columns beyond the matrix, the last tile not whole
    (9000, 260, 1024),     # entry points, columns beyond the matrix
    (9000, 256, 1024),     # entry points, whole blocks of columns
    (16000, 2048, 16),     # eight rows a bin
])
@pytest.mark.parametrize("ids", ["spread", "sorted", "one", "few", "invalid", "most", "skewed", "padded"])
def test_grouped_gather(V, H, th, ids):
    import comp_inference_b200 as ci
    g = torch.Generator("cuda").manual_seed(V)
    W = (torch.randn(V, H, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    c = ci.compress_weight_cuda(W, th, 32)
    m = ci.RansEmbedding(V, H, c["tile_height"], 32).load_compressed(c).prepare()
    n = 4096 if ids != "most" else 9001                 # more than one launch takes, whatever takes the rest
    i = torch.randint(0, V, (n,), generator=g, device="cuda")
    if ids == "sorted":
        i = i.sort().values
    elif ids == "one":
        i[:] = V - 1                                    # one bin of all ids
    elif ids == "few":
        i = i % 200 * (V // 200)                        # bins of one row and 20 ids, and of several
    elif ids == "skewed":                               # several bins of more than 128 ids, of one row and of many
        i = (torch.rand(n, generator=g, device="cuda") * math.log(V)).exp().long() - 1
    elif ids == "padded":                               # two bins of more, in runs and in between
        i[:1300], i[2000::2] = 0, V - 1
    elif ids == "invalid":
        i[::3], i[1::7] = -1, V                         # a bin of ids outside the table
    out = m(i)
    ok = (i >= 0) & (i < V)
    want = torch.where(ok[:, None], W[i.clamp(0, V - 1)], torch.zeros((), dtype=torch.bfloat16, device="cuda"))
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("V,H,th,n,groups,single", [
    (32000, 4096, 16, 4096, 1, 0),
    (32000, 4096, 16, 4097, 0, 1),      # one more than a launch takes: what groups gain is less than a second launch costs
    (32000, 4096, 16, 8200, 0, 1),
    (16000, 2048, 16, 8192, 2, 0),      # two whole launches
    (4000, 512, 64, 4100, 1, 1),        # a rest too small for groups
    (5001, 1100, 128, 9001, 3, 0),      # a rest that is not
    (4001, 1100, 128, 4100, 0, 1),      # too few bins
])
def test_batches_of_many_launches(V, H, th, n, groups, single):
    import comp_inference_b200 as ci
    g = torch.Generator("cuda").manual_seed(n)
    W = (torch.randn(V, H, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    c = ci.compress_weight_cuda(W, th, 32)
    m = ci.RansEmbedding(V, H, c["tile_height"], 32).load_compressed(c).prepare()
    i = torch.randint(0, V, (n,), generator=g, device="cuda")
    assert torch.equal(m(i).view(torch.int16), W[i].view(torch.int16))
    launched = captured_kernels(lambda: m(i))
    assert (launched.count("k_embedding_group"), launched.count("k_embedding4")) == (groups, single)
