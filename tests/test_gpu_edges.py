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
                                      (2048, 8192, 128, 16), (2056, 8196, 128, 11), (4096, 8192, 64, 5),
                                      # K ends inside a group of four rows, in every quarter of a pair of tiles
                                      (2050, 4096, 128, 1), (2113, 4099, 128, 4), (2177, 4097, 128, 2), (2247, 4096, 128, 16),
                                      (1027, 64, 1024, 1), (1537, 32, 1024, 3), (3070, 40, 1024, 9), (4095, 64, 512, 1)])
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


# every split of the one-pass encoder (one / two columns a lane, one / two halves), odd and ragged sides, streams whose
# length is no multiple of four symbols' worth of rows, a plane of one symbol, symbols of frequency one
@pytest.mark.parametrize("K,N,th", [(2048, 4800, 64), (2050, 4800, 64), (1100, 2432, 128), (1000, 77, 128), (16, 1, 16),
                                    (33, 64, 16), (2049, 130, 1024), (40, 62, 32)])
@pytest.mark.parametrize("kind", ["normal", "wide", "constant"])
def test_one_pass_encoder_matches_oracle(K, N, th, kind):
    import numpy as np
    import comp_inference_b200 as ci
    from oracle import oracle as O
    g = torch.Generator().manual_seed(K * 31 + N)
    W = {"normal": lambda: torch.randn(K, N, generator=g) * 0.02,
         "wide": lambda: torch.randn(K, N, generator=g) * 2.0 ** torch.randint(-100, 100, (K, N), generator=g),
         "constant": lambda: torch.full((K, N), 1.5)}[kind]().to(torch.bfloat16)
    c = ci.compress_weight_cuda(W.cuda(), th, 32)
    o = O.compress_bf16(W.view(torch.uint16).numpy(), c["tile_height"], c["tile_width"])
    host = lambda name: c[name].cpu().view(torch.uint8).numpy()
    for name, want in (("rans_exp_stream", o.stream), ("rans_exp_states", o.states), ("rans_exp_tables", o.tables),
                       ("rans_exp_slot_map", o.slot_map), ("rans_exp_tile_offsets", o.tile_offsets),
                       ("rans_exp_tile_max_lens", o.tile_max_lens), ("rans_man_raw", o["mantissa"])):
        assert np.array_equal(host(name), np.ascontiguousarray(want).view(np.uint8).reshape(-1)), name
    plane, _ = ci.extract_exp_and_mantissa(W.cuda())
    r = ci.ccore.RansManager().compress_tiled(plane, c["exponent_freqs"], c["exponent_cdf"], th, 32)
    assert torch.equal(r.stream, c["rans_exp_stream"].cpu()) and torch.equal(r.output_sizes.view(torch.int32),
                                                                            c["output_sizes"].cpu().view(torch.int32))


# stored-transposed linear: rows that end inside a tile / a group of four tiles, a last column block that ends inside a
# lane's quad, one and several passes over the activation rows, tall tiles (fewer sums fit), runs that cross groups
@pytest.mark.parametrize("V,H,th,M", [(512, 64, 128, 1), (2000, 100, 128, 2), (1111, 33, 64, 3), (333, 250, 16, 8),
                                      (5000, 128, 1024, 1), (4099, 96, 1024, 5), (777, 1030, 256, 9), (16000, 512, 128, 1),
                                      (40, 16, 32, 17)])
def test_transposed_linear_edges(V, H, th, M):
    import comp_inference_b200 as ci
    from comp_inference_b200 import _lib
    W = _weight(V, H)
    c = ci.compress_weight_cuda(W, th, 32)
    x = torch.randn(M, H, generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).cuda()
    bias = torch.randn(V, generator=torch.Generator().manual_seed(V)).to(torch.bfloat16).cuda()
    args = (c["rans_exp_stream"], c["rans_exp_states"], c["rans_exp_tables"], c["rans_exp_slot_map"], (V, H),
            c["rans_exp_tile_offsets"], c["rans_exp_tile_max_lens"], c["tile_height"], c["tile_width"], c["rans_man_raw"])
    y = ci.fused_rans_linear_transposed_triton(x, *args, bias=bias)
    assert _close(y, x.float() @ W.float().t() + bias.float())
    assert torch.equal(y, ci.fused_rans_linear_transposed_triton(x, *args, bias=bias))   # workspace left clean, same order
    assert _lib.kernel_status(x.device) == 0


# stand-alone decoder: a last tile row that is not whole, odd widths, tall tiles with one window, both planes
@pytest.mark.parametrize("K,N,th", [(100, 64, 128), (2050, 96, 1024), (4096, 160, 1024), (1111, 77, 128), (513, 30, 256),
                                    (48, 41, 16), (640, 2050, 64)])
def test_decoder_edges(K, N, th):
    import comp_inference_b200 as ci
    W = _weight(K, N)
    c = ci.compress_weight_cuda(W, th, 32)
    args = (c["rans_exp_stream"], c["rans_exp_states"], c["rans_exp_tables"], c["rans_exp_slot_map"])
    tile = (c["rans_exp_tile_offsets"], c["rans_exp_tile_max_lens"], c["tile_height"], c["tile_width"])
    w = ci.rans_decompress_bf16(*args, (K, N), *tile, c["rans_man_raw"])
    assert torch.equal(w.view(torch.int16), W.view(torch.int16))
    plane = ci.rans_decomp_triton_tiled(*args, (K, N), *tile)
    assert torch.equal(plane, ci.extract_exp_and_mantissa(W)[0])


# two streams a lane (few tiles: short and missing bottom halves, odd widths and rows, several rounds of tall tiles) and its
# neighbour, four streams at sizes with many tiles
@pytest.mark.parametrize("K,N,th", [(700, 33, 1024), (520, 130, 1024), (512, 64, 1024), (513, 4099, 1024), (8200, 1186, 2048),
                                    (16, 31, 16), (4097, 2014, 128), (2111, 8222, 64), (4096, 4100, 128)])
def test_decoder_few_and_many_tiles(K, N, th):
    test_decoder_edges(K, N, th)


# row gather: every row of small tables (each position inside a half tile), ids outside, one id, more ids than warps,
# tall tiles (one window per warp), odd widths
@pytest.mark.parametrize("V,H,th,n", [(96, 128, 16, 300), (300, 4096, 16, 1), (257, 100, 128, 257), (3000, 64, 1024, 500),
                                      (2048, 1030, 1024, 40), (640, 320, 64, 5000), (64, 33, 32, 70)])
def test_embedding_edges(V, H, th, n):
    import comp_inference_b200 as ci
    W = _weight(V, H)
    c = ci.compress_weight_cuda(W, th, 32)
    m = ci.RansEmbedding(V, H, c["tile_height"], c["tile_width"]).load_compressed(c).prepare()
    ids = torch.arange(n, device="cuda") % (V + 2) - 1
    want = torch.where(((ids >= 0) & (ids < V))[:, None], W[ids.clamp(0, V - 1)].float(), torch.zeros((), device="cuda"))
    assert torch.equal(m(ids).float(), want)
    assert torch.equal(m(ids.view(1, -1).to(torch.int32))[0].float(), want)


# prompts through the module: sizes whose rows the library cannot take aligned, tall tiles entered at entry points
@pytest.mark.parametrize("K,N,th,M", [(1000, 776, 128, 20), (1001, 776, 128, 33), (1000, 777, 64, 17), (2305, 131, 1024, 65),
                                      (3072, 512, 512, 40), (1024, 96, 1024, 18)])
def test_prompt_edges(K, N, th, M):
    import comp_inference_b200 as ci
    W = _weight(K, N)
    c = ci.compress_weight_cuda(W, th, 32)
    m = ci.RansLinear(K, N, c["tile_height"], c["tile_width"], has_bias=True)
    m.bias = torch.randn(N, generator=torch.Generator().manual_seed(N)).to(torch.bfloat16).cuda()
    m.load_compressed(c).prepare()
    x = torch.randn(2, M, K, generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).cuda()
    for x in (x, x[:1, :, :].transpose(0, 1)):
        y = m(x)
        assert y.shape == (*x.shape[:-1], N) and y.is_contiguous()
        assert _close(y, x.float() @ W.float() + m.bias.float())


# end of a greedy step: ties, NaN, infinities, widths that are no multiple of eight, one and several sequences
@pytest.mark.parametrize("B,V", [(1, 32000), (3, 101), (8, 4096), (5, 1), (2, 50257)])
def test_greedy_step(B, V):
    from comp_inference_b200 import ops
    logits = torch.randn(B, V, generator=torch.Generator().manual_seed(V)).to(torch.bfloat16)
    logits[0, V // 2:] = logits[0].max()
    if B > 1:
        logits[1, V // 3] = float("inf")
        logits[B - 1] = -logits[B - 1].abs() if V > 1 else 0.0
        logits[B - 1, V - 1] = -0.0
    if B > 2:
        logits[2, V // 5] = float("nan")
    logits = logits.cuda()
    tok, out = torch.zeros(B + 1, dtype=torch.int64, device="cuda"), torch.zeros(B + 1, 4, dtype=torch.int64, device="cuda")
    pos, steps = torch.full((1,), 7, device="cuda"), torch.zeros(1, dtype=torch.int64, device="cuda")
    ticket = torch.zeros(1, dtype=torch.int32, device="cuda")
    want = logits.argmax(-1)
    for i in range(1, 4):
        ops.greedy_step(logits, tok, pos, steps, out, ticket)
        assert torch.equal(tok[:B], want) and torch.equal(out[:B, i], want)
        assert int(pos) == 7 + i and int(steps) == i and int(ticket) == 0
    assert int(tok[B]) == 0 and int(out[B].sum()) == 0


# columns beyond N run along with others: one to three left in a lane's quad, lanes and tiles without any; whole and
# ragged K, with and without entry points
@pytest.mark.parametrize("K,N,th,M", [(8192, 4097, 128, 1), (8200, 4098, 64, 9), (8192, 4115, 128, 16), (2048, 35, 1024, 2),
                                      (2049, 61, 1024, 5), (4100, 2020, 1024, 1)])
def test_column_edges(K, N, th, M):
    import comp_inference_b200 as ci
    W = _weight(K, N)
    c = ci.compress_weight_cuda(W, th, 32)
    m = ci.RansLinear(K, N, c["tile_height"], c["tile_width"]).load_compressed(c).prepare()
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(K)).to(torch.bfloat16).cuda()
    assert _close(m(x), x.float() @ W.float())
    test_decoder_edges(K, N, th)


# prompts whose buffers the staged decoders do not take (slices of a larger buffer): odd sizes are decoded into padded rows all the same
@pytest.mark.parametrize("K,N,th", [(1000, 776, 128), (1000, 777, 128), (515, 131, 1024)])
@pytest.mark.parametrize("name", ["rans_exp_stream", "rans_exp_states", "rans_man_raw"])
def test_prompt_from_unaligned_buffers(K, N, th, name):
    import comp_inference_b200 as ci
    W = _weight(K, N)
    c = ci.compress_weight_cuda(W, th, 32)
    t = c[name]
    c[name] = torch.empty(t.numel() + 1, dtype=torch.uint8 if t.dtype == torch.uint8 else torch.int32, device="cuda").view(t.dtype)[1:]
    c[name].copy_(t)
    m = ci.RansLinear(K, N, c["tile_height"], c["tile_width"]).load_compressed(c).prepare()
    x = torch.randn(20, K, generator=torch.Generator().manual_seed(N)).to(torch.bfloat16).cuda()
    for rows in (20, 3):
        assert _close(m(x[:rows]), x[:rows].float() @ W.float())


# tall tiles of incompressible exponents: a window of the staged decoder does not fit, so there are no entry points
@pytest.mark.parametrize("K,N,th", [(4096, 64, 4096), (4100, 40, 4096)])
def test_tiles_too_deep_for_entry_points(K, N, th):
    import comp_inference_b200 as ci
    g = torch.Generator().manual_seed(K)
    W = (torch.randn(K, N, generator=g) * 2.0 ** torch.randint(-100, 1, (K, N), generator=g)).to(torch.bfloat16).cuda()
    c = ci.compress_weight_cuda(W, th, 32)
    assert c["tile_height"] == th and int(c["rans_exp_tile_max_lens"].view(torch.int32).max()) > 1550
    m = ci.RansLinear(K, N, th, 32).load_compressed(c).prepare()
    x = torch.randn(20, K, generator=g).to(torch.bfloat16).cuda()
    for rows in (1, 20):
        assert _close(m(x[:rows]), x[:rows].float() @ W.float())
    e = ci.RansEmbedding(K, N, th, 32).load_compressed(c).prepare()
    ids = torch.tensor([0, K // 2 - 1, K // 2, K - 1], device="cuda")
    assert torch.equal(e(ids), W[ids])


# the workspace of the size that the library names is all that a call touches: activations reordered behind the partial sums,
# fewer rows than a group of four, workspaces that end off a 256-byte boundary
@pytest.mark.parametrize("K,N,M", [(1, 28419, 15), (5, 28419, 15), (9, 28419, 15), (1, 28419, 13), (1001, 28419, 15), (18, 28419, 16)])
def test_linear_stays_inside_its_workspace(K, N, M):
    from comp_inference_b200 import _lib
    lib = _lib.load()
    W = _weight(K, N)
    stream, states, _, tables, slot_map, offsets, lens, man, *_ = _lib.host().compress(W, 16, 32, False)
    w, keep = _lib.tiled_weight(stream, states, tables, slot_map, offsets, lens, man, K, N, 16, 32, want_max=True)
    assert lib.ci_linear_route(w, M) == 2
    n = lib.ci_linear_workspace_bytes(M, N, K, 16)
    ws = torch.zeros(n + 4096, dtype=torch.uint8, device="cuda")
    ws[n:] = 0xA5
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).cuda()
    y = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    _lib.check(lib.ci_linear(w, _lib.ptr(x), K, M, None, _lib.ptr(y), N, _lib.ptr(ws), n, 0, _lib.stream()))
    assert _close(y, x.float() @ W.float())
    assert bool((ws[n:] == 0xA5).all())


# the encoder's sign+mantissa bytes to an odd address, at sizes where a lane takes two columns and one
@pytest.mark.parametrize("K,N", [(2048, 4800), (1000, 78)])
def test_encoder_to_an_odd_address(K, N):
    import ctypes as C
    import comp_inference_b200 as ci
    from comp_inference_b200 import _lib
    lib = _lib.load()
    W = _weight(K, N)
    c = ci.compress_weight_cuda(W, 64, 32)
    tiles, want = -(-K // 64) * -(-N // 32), c["rans_man_raw"]
    man = torch.zeros(want.numel() + 1, dtype=torch.uint8, device="cuda")[1:]
    u32 = lambda n: torch.empty(n, dtype=torch.int32, device="cuda")
    states, sizes, offsets, lens, tables = u32(tiles * 64), u32(tiles * 64), u32(tiles), u32(tiles), u32(256)
    slot_map, freqs, cdf = torch.empty(4096, dtype=torch.uint8, device="cuda"), torch.empty(256, dtype=torch.uint16), torch.empty(256, dtype=torch.uint16)
    n_scratch, n = lib.ci_compress_scratch_bytes(K, N, 64, 32), C.c_uint64(0)
    scratch = torch.empty(n_scratch, dtype=torch.uint8, device="cuda")
    _lib.check(lib.ci_compress_bf16(_lib.ptr(W), K, N, 64, 32, *map(_lib.ptr, (man, states, sizes, offsets, lens, tables, slot_map, scratch)),
                                    n_scratch, _lib.ptr(freqs), _lib.ptr(cdf), None, C.byref(n), _lib.stream()))
    assert torch.equal(man, want) and n.value == c["rans_exp_stream"].numel()
    assert torch.equal(states, c["rans_exp_states"].view(torch.int32))


# depths left over in the output array, in as many tiles as one block clears, one more, and several blocks' worth
@pytest.mark.parametrize("K,N", [(8176, 1024), (8192, 1024), (16 * 1171, 32 * 43)])
def test_encoder_clears_the_depths(K, N):
    import ctypes as C
    import comp_inference_b200 as ci
    from comp_inference_b200 import _lib
    lib = _lib.load()
    W = _weight(K, N)
    c = ci.compress_weight_cuda(W, 16, 32)
    tiles, want = -(-K // 16) * -(-N // 32), c["rans_exp_tile_max_lens"].view(torch.int32)
    assert 0 < int(want.max()) <= 16
    u32 = lambda n: torch.full((n,), 0x7FFFFFFF, dtype=torch.int32, device="cuda")
    man = torch.empty_like(c["rans_man_raw"])
    states, sizes, offsets, lens, tables = u32(tiles * 64), u32(tiles * 64), u32(tiles), u32(tiles), u32(256)
    slot_map, freqs, cdf = torch.empty(4096, dtype=torch.uint8, device="cuda"), torch.empty(256, dtype=torch.uint16), torch.empty(256, dtype=torch.uint16)
    n_scratch, n = lib.ci_compress_scratch_bytes(K, N, 16, 32), C.c_uint64(0)
    scratch = torch.empty(n_scratch, dtype=torch.uint8, device="cuda")
    _lib.check(lib.ci_compress_bf16(_lib.ptr(W), K, N, 16, 32, *map(_lib.ptr, (man, states, sizes, offsets, lens, tables, slot_map, scratch)),
                                    n_scratch, _lib.ptr(freqs), _lib.ptr(cdf), None, C.byref(n), _lib.stream()))
    assert torch.equal(lens, want) and n.value == c["rans_exp_stream"].numel()
    plane, _ = ci.extract_exp_and_mantissa(W)
    lens.fill_(0x7FFFFFFF)
    _lib.check(lib.ci_compress_plane(_lib.ptr(plane), K, N, _lib.ptr(freqs), _lib.ptr(cdf), 16, 32, *map(
        _lib.ptr, (states, sizes, offsets, lens, tables, slot_map, scratch)), n_scratch, C.byref(n), _lib.stream()))
    assert torch.equal(lens, want) and n.value == c["rans_exp_stream"].numel()


# threads that compress one after the other: each has a landing place of its own, given back when it ends
def test_encoder_from_threads_that_end():
    import threading
    import comp_inference_b200 as ci
    W = _weight(256, 64)
    want, got = ci.compress_weight_cuda(W, 64, 32), []
    for _ in range(8):
        t = threading.Thread(target=lambda: got.append(ci.compress_weight_cuda(W, 64, 32)))
        t.start()
        t.join()
    assert len(got) == 8 and all(torch.equal(c["rans_exp_stream"], want["rans_exp_stream"]) for c in got)


# one symbol only: a last tile row too short to emit a byte, below tiles that have some, entered at entry points
@pytest.mark.parametrize("K,N,th", [(342, 64, 256), (342, 2647, 256), (1100, 33, 1024), (3072 + 40, 96, 1024)])
def test_entry_points_of_tiles_without_bytes(K, N, th):
    import comp_inference_b200 as ci
    from comp_inference_b200 import _lib
    W = torch.full((K, N), 1.5, dtype=torch.bfloat16, device="cuda")
    c = ci.compress_weight_cuda(W, th, 32)
    depths = c["rans_exp_tile_max_lens"].view(torch.int32)
    assert int(depths.min()) == 0 and int(depths.max()) > 0
    m = ci.RansLinear(K, N, th, 32).load_compressed(c).prepare()
    h = ci.RansLMHead(N, K, th, 32, fast_twin=False).load_compressed(c).prepare()
    for M in (1, 9, 20):
        x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).cuda()
        assert _close(m(x), x.float() @ W.float())
        xh = x.repeat(1, -(-N // K))[:, :N]
        assert _close(h(xh), xh.float() @ W.float().t())
    ids = torch.tensor([0, th // 2, th, K - 1], device="cuda")
    assert torch.equal(ci.RansEmbedding(K, N, th, 32).load_compressed(c).prepare()(ids), W[ids])
    assert _lib.kernel_status(W.device) == 0
