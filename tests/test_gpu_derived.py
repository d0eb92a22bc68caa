"""What is derived from a weight's arrays and kept between calls (decode table, deepest tile, entry points into tall tiles)
follows the arrays."""
import pytest
import torch

from conftest import make_weight

pytestmark = pytest.mark.gpu

ARRAYS = ("rans_exp_stream", "rans_exp_states", "rans_exp_tables", "rans_exp_slot_map", "rans_exp_tile_offsets",
          "rans_exp_tile_max_lens", "rans_man_raw")
K, N, TH, M = 2048, 96, 1024, 2


def _two_weights():
    """Two weights whose packages differ in stream, states and sign+mantissa bytes only: the columns of the second are the
    first's, swapped in pairs, so every tile has the same streams in another order."""
    import comp_inference_b200 as ci
    a = make_weight(K, N, 5)
    b = a.view(K, N // 2, 2).flip(-1).reshape(K, N)
    ca, cb = (ci.compress_weight_cuda(w.cuda(), TH, 32) for w in (a, b))
    for name in ARRAYS[2:6]:
        assert torch.equal(ca[name].view(torch.uint8), cb[name].view(torch.uint8)), name
    assert ca["rans_exp_stream"].numel() == cb["rans_exp_stream"].numel()
    assert not torch.equal(ca["rans_exp_states"].view(torch.int32), cb["rans_exp_states"].view(torch.int32))
    return a.cuda(), ca, b.cuda(), cb


def _call(kind, c, x, ids):
    import comp_inference_b200 as ci
    args = [c[n] for n in ARRAYS[:4]] + [(K, N), c["rans_exp_tile_offsets"], c["rans_exp_tile_max_lens"], TH, 32, c["rans_man_raw"]]
    if kind == "linear":
        return ci.fused_rans_linear_triton(x, *args)
    if kind == "transposed":
        return ci.fused_rans_linear_transposed_triton(x[:, :N], *args)
    return ci.fused_rans_embedding_triton(ids, *args)


def _right(kind, y, w, x, ids):
    if kind == "embedding":
        return torch.equal(y, w[ids])
    ref = x.float() @ w.float() if kind == "linear" else x[:, :N].float() @ w.float().t()
    return float((y.float() - ref).abs().max() / ref.abs().max()) <= 1e-2


def _inputs():
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(7)).to(torch.bfloat16).cuda()
    return x, torch.randint(0, K, (50,), generator=torch.Generator().manual_seed(8)).cuda()


@pytest.mark.parametrize("kind", ["linear", "transposed", "embedding"])
@pytest.mark.parametrize("how", ["other tensors", "overwritten"])
def test_functional_calls_follow_the_streams(kind, how):
    wa, ca, wb, cb = _two_weights()
    x, ids = _inputs()
    assert _right(kind, _call(kind, ca, x, ids), wa, x, ids)
    if how == "other tensors":                          # a second weight that shares the arrays it can share
        cb = dict(cb, **{n: ca[n] for n in ARRAYS[2:6]})
        assert _right(kind, _call(kind, cb, x, ids), wb, x, ids)
    else:
        for n in ("rans_exp_stream", "rans_exp_states", "rans_man_raw"):
            ca[n].copy_(cb[n])
        assert _right(kind, _call(kind, ca, x, ids), wb, x, ids)


def _module(kind, c):
    import comp_inference_b200 as ci
    m = {"linear": lambda: ci.RansLinear(K, N, TH, 32), "embedding": lambda: ci.RansEmbedding(K, N, TH, 32),
         "transposed": lambda: ci.RansLMHead(N, K, TH, 32, fast_twin=False), "twin": lambda: ci.RansLMHead(N, K, TH, 32)}[kind]()
    return m.load_compressed({n: c[n].clone() for n in ARRAYS}).prepare()


@pytest.mark.parametrize("kind", ["linear", "embedding", "transposed", "twin"])
@pytest.mark.parametrize("how", ["overwritten", "replaced"])
@pytest.mark.parametrize("what", ["streams", "tables"])
def test_modules_follow_their_buffers(kind, how, what):
    wa, ca, wb, cb = _two_weights()
    changed = ("rans_exp_stream", "rans_exp_states", "rans_man_raw")
    if what == "tables":                                # the same bytes read as exponents one higher: twice the weight
        wb, changed = wa * 2, ARRAYS[2:4]
        cb = dict(ca, rans_exp_tables=ca["rans_exp_tables"].view(torch.int32).roll(1).view(torch.uint32),
                  rans_exp_slot_map=ca["rans_exp_slot_map"] + 1)
    x, ids = _inputs()
    m = _module(kind, ca)

    def right(w):
        if kind == "embedding":
            return _right(kind, m(ids), w, x, ids)
        if kind == "linear":                            # and as a prompt: decoded first
            xl = x.repeat(10, 1)
            return _right(kind, m(x), w, x, ids) and _right(kind, m(xl), w, xl, ids)
        return _right("transposed", m(x[:, :N].contiguous()), w, x, ids)

    assert right(wa)
    if how == "replaced":
        m.load_compressed({n: cb[n].clone() for n in changed})
    else:
        for n in changed:
            getattr(m, n).copy_(cb[n])
    assert right(wb)


def _captured(fn):
    """fn captured on a stream of its own, replayed once: (graph, result)."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        y = fn()
    y.zero_()
    graph.replay()
    torch.cuda.synchronize()
    return graph, y


@pytest.mark.parametrize("kind", ["linear", "transposed", "embedding", "prompt"])
@pytest.mark.parametrize("before", ["nothing", "decoded", "called", "overwritten"])
def test_first_call_under_capture(kind, before):
    """Nothing is read back while a stream captures, and what a capture makes is not kept for calls outside it."""
    import comp_inference_b200 as ci
    from comp_inference_b200 import _lib
    wa, ca, wb, cb = _two_weights()
    x, ids = _inputs()
    if kind == "prompt":
        x = x.repeat(10, 1)
        m = ci.RansLinear(K, N, TH, 32).load_compressed(ca)
        call, kind = lambda: m(x), "linear"
    else:
        call = lambda: _call(kind, ca, x, ids)
    w = wa
    if before in ("decoded", "overwritten"):
        args = [ca[n] for n in ARRAYS[:4]] + [(K, N), ca["rans_exp_tile_offsets"], ca["rans_exp_tile_max_lens"], TH, 32, ca["rans_man_raw"]]
        assert torch.equal(ci.rans_decompress_bf16(*args), w)
    if before in ("called", "overwritten"):
        assert _right(kind, call(), w, x, ids)
    if before == "overwritten":
        w = wb
        for n in ("rans_exp_stream", "rans_exp_states", "rans_man_raw"):
            ca[n].copy_(cb[n])
    graph, y = _captured(call)
    assert _right(kind, y, w, x, ids)
    assert _right(kind, call(), w, x, ids)
    del graph, y
    assert _right(kind, call(), w, x, ids)
    assert _lib.kernel_status(x.device) == 0


@pytest.mark.parametrize("layout", ["tiled", "dense"])
def test_table_prepared_on_another_stream(layout):
    """A decode table made by a call on one stream is whole for a call on another one, which has waited for the arrays only."""
    import comp_inference_b200 as ci
    w = make_weight(256, 64, 5)
    c = ci.compress_weight_cuda(w.cuda(), 64, 32, uncoalesced_interleaving=layout == "dense")
    fn = ci.fused_rans_embedding_triton if layout == "tiled" else ci.fused_rans_embedding_triton_uncoalesced
    places = ("rans_exp_tile_offsets", "rans_exp_tile_max_lens") if layout == "tiled" else ("rans_exp_stream_offsets", "output_sizes")
    args = [c[n] for n in ARRAYS[:4]] + [(256, 64), *(c[n] for n in places), 64, 32, c["rans_man_raw"]]
    tables, slot_map = args[2], args[3]
    ids = torch.arange(256, device="cuda")
    fn(ids, *args[:2], tables.clone(), slot_map.clone(), *args[4:])      # kernels are loaded: loading one waits for the device
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        if layout == "tiled":                           # everything known, then the tables change: exponents one higher
            assert torch.equal(fn(ids, *args), w.cuda())
            tables.copy_(tables.view(torch.int32).roll(1).view(torch.uint32))
            slot_map.add_(1)
            w = w * 2
        stale = torch.full((4096,), -1, dtype=torch.int32, device="cuda")    # what the table's memory may hold before it is made
        del stale
        ready = a.record_event()
        torch.cuda._sleep(100_000_000)
        fn(ids, *args)
    b.wait_event(ready)
    with torch.cuda.stream(b):
        y = fn(ids, *args)
    torch.cuda.synchronize()
    assert torch.equal(y, w.cuda())


@pytest.mark.parametrize("kind", ["linear", "transposed"])
def test_entry_points_that_contradict_the_depths_are_reported(kind):
    """A write that no version counter sees leaves entry points behind which reach beyond a tile's byte block (here: by one
    row, inside the stream): nothing is read there, and the status word says so."""
    import comp_inference_b200 as ci
    wa, ca, _, _ = _two_weights()
    x, ids = _inputs()
    assert _right(kind, _call(kind, ca, x, ids), wa, x, ids)
    ci.check_status()
    ca["rans_exp_tile_max_lens"].view(torch.int32).data.sub_(1)
    _call(kind, ca, x, ids)
    with pytest.raises(RuntimeError, match="status 2"):
        ci.check_status()
    ci.check_status()


@pytest.mark.parametrize("k,n,th,rows,route", [(1024, 256, 256, 1, 2), (1024, 256, 256, 16, 2), (1024, 256, 128, 1, 1), (4096, 2048, 128, 1, 2),
                                               (1024, 256, 256, 17, 3)])
def test_route_of_a_module_counts_its_entry_points(k, n, th, rows, route):
    import comp_inference_b200 as ci
    m = ci.RansLinear(k, n, th, 32).load_compressed(ci.compress_weight_cuda(make_weight(k, n, 5).cuda(), th, 32)).prepare()
    assert m._native().route(rows) == route             # 1: two streams a lane, 2: four, 3: decode-GEMM (ci_linear_route)


@pytest.mark.parametrize("kind", ["linear", "transposed", "embedding", "module"])
@pytest.mark.parametrize("th", [1024, 128])
def test_a_weight_written_by_the_kernel_before(kind, th):
    """The arrays may be products of the kernel that comes right before a call, which starts to read the weight early."""
    import comp_inference_b200 as ci
    a = make_weight(K, N, 5)
    ws = [a.cuda(), a.view(K, N // 2, 2).flip(-1).reshape(K, N).cuda()]
    cs = [ci.compress_weight_cuda(w, th, 32) for w in ws]
    x, ids = _inputs()
    c = {n: cs[0][n].clone() for n in ARRAYS}
    m = ci.RansLinear(K, N, th, 32).load_compressed(c)
    args = [c[n] for n in ARRAYS[:4]] + [(K, N), c["rans_exp_tile_offsets"], c["rans_exp_tile_max_lens"], th, 32, c["rans_man_raw"]]
    call = {"linear": lambda: ci.fused_rans_linear_triton(x, *args), "module": lambda: m(x),
            "transposed": lambda: ci.fused_rans_linear_transposed_triton(x[:, :N], *args),
            "embedding": lambda: ci.fused_rans_embedding_triton(ids, *args)}[kind]
    out = []
    for i in range(20):
        for n, dt in (("rans_exp_stream", torch.uint8), ("rans_man_raw", torch.uint8), ("rans_exp_states", torch.int32)):
            torch.add(cs[i % 2][n].view(dt), 0, out=c[n].view(dt))      # a kernel, where copy_ would be a copy
        out.append(call())
    for i, y in enumerate(out):
        assert _right("linear" if kind == "module" else kind, y, ws[i % 2], x, ids)


@pytest.mark.parametrize("kind", ["linear", "transposed", "prompt", "dense"])
def test_graphs_replayed_in_another_order_than_captured(kind):
    """Two graphs captured on one stream that no call ran on before, in a pool they share with others: neither counts on
    what the other would have zeroed."""
    import comp_inference_b200 as ci
    from comp_inference_b200 import _lib
    wa, ca, _, _ = _two_weights()
    x, _ = _inputs()
    if kind == "dense":
        c = ci.compress_weight_cuda(wa, 64, 32, uncoalesced_interleaving=True)
        call = lambda: ci.fused_rans_linear_triton_uncoalesced(
            x, c["rans_exp_stream"], c["rans_exp_states"], c["rans_exp_tables"], c["rans_exp_slot_map"], (K, N),
            c["rans_exp_stream_offsets"], c["output_sizes"], c["tile_height"], 32, c["rans_man_raw"])
    elif kind == "prompt":
        x = x.repeat(10, 1)
        m = ci.RansLinear(K, N, TH, 32).load_compressed(ca).prepare()
        call = lambda: m(x)
    else:
        call = lambda: _call(kind, ca, x, None)
    kind = "linear" if kind in ("dense", "prompt") else kind
    assert _right(kind, call(), wa, x, None)
    used = {key[1] for key in _lib._workspaces}
    side = next(s for s in (torch.cuda.Stream() for _ in range(64)) if s.cuda_stream not in used)
    pool, graphs = torch.cuda.graph_pool_handle(), []

    def capture(fn):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side, pool=pool):
            y = fn()
        return g, y

    before, _ = capture(lambda: torch.full((64 << 20,), 255, dtype=torch.uint8, device="cuda").sum())
    before.replay()                                     # what the pool's memory holds
    torch.cuda.synchronize()
    graphs = [capture(call), capture(call)]
    for g, y in reversed(graphs):
        g.replay()
        torch.cuda.synchronize()
        assert _right(kind, y, wa, x, None)
    with torch.cuda.stream(side):
        y = call()
    torch.cuda.synchronize()
    assert _right(kind, y, wa, x, None)
    assert _lib.kernel_status(x.device) == 0
