"""The work that users of this framework have it do, as a list of measurable cases.

Shapes are those of the repository's benchmark and tests (the linears, embedding table and head of a Llama-2-7B
sized model, their tensor-parallel shards) and generic ones between them.  Weights are seeded N(0, 0.02) bf16,
compressed by the framework itself; a tile height of 1024 is the format's default, 128 / 64 / 16 are the heights
the benchmark, the tensor-parallel loader and the whole-model run store.

    linear      y = x . W (+ bias) through RansLinear ("module") or fused_rans_linear_triton with its default
                arguments ("function"); up to 16 rows are decode steps, more are prompts
    block       the linears of one decoder block in order, q|k|v and gate|up concatenated, one token batch
    head        logits from a table stored [V, H] (tied head), fused_rans_linear_transposed_triton
    embedding   RansEmbedding row gather
    decompress  a whole weight back to bf16
    compress    a bf16 weight to the tiled package arrays
    step        a captured decode step of LlamaGreedyRunner: embedding, decoder layers with attention over a
                filled cache, head
"""
import math
from types import SimpleNamespace

import torch
import torch.nn as nn

import comp_inference_b200 as ci
from comp_inference_b200.generation import LlamaGreedyRunner

HEAD_DIM = 128


def listed():
    return [
        # one rank's o_proj shard at eight ranks, one token: the smallest call, launch latency and host time count
        {"name": "linear_shard_b1", "kind": "linear", "api": "module", "K": 512, "N": 4096, "tile": 64, "M": 1, "bias": False},
        # a package written with the format's default tile, one token at a time
        {"name": "linear_default_tile_b1", "kind": "linear", "api": "module", "K": 4096, "N": 4096, "tile": 1024, "M": 1,
         "bias": False},
        # the functional call as the original library's users write it, ragged sizes, a few sequences at once
        {"name": "linear_function_b5", "kind": "linear", "api": "function", "K": 5504, "N": 4100, "tile": 128, "M": 5,
         "bias": True},
        # the benchmark's workload: one decoder block, one token; and a full batch of sequences
        {"name": "block_b1", "kind": "block", "hidden": 4096, "ffn": 11008, "tile": 128, "M": 1},
        {"name": "block_b16", "kind": "block", "hidden": 4096, "ffn": 11008, "tile": 128, "M": 16},
        # a short prompt of odd length, and the prompt pass of a large batch
        {"name": "linear_prompt_77", "kind": "linear", "api": "module", "K": 4096, "N": 11008, "tile": 128, "M": 77,
         "bias": False},
        {"name": "linear_prompt_2048", "kind": "linear", "api": "module", "K": 4096, "N": 22016, "tile": 128, "M": 2048,
         "bias": False},
        # logits of one token from the embedding table as it is stored
        {"name": "head_stored_b1", "kind": "head", "V": 32000, "H": 4096, "tile": 128, "M": 1},
        # the embedding of a prompt batch
        {"name": "embedding_4096", "kind": "embedding", "V": 32000, "H": 4096, "tile": 16, "ids": 4096},
        # a default-tile weight restored for a dense consumer; a weight compressed when a package is written
        {"name": "decompress_default_tile", "kind": "decompress", "K": 4096, "N": 11008, "tile": 1024},
        {"name": "compress", "kind": "compress", "K": 4096, "N": 11008, "tile": 128},
        # a serving step of eight sequences, two layers of a model
        {"name": "step_b8", "kind": "step", "hidden": 4096, "ffn": 11008, "vocab": 32000, "layers": 2, "tile": 128,
         "batch": 8, "context": 1024},
    ]


def _size(rng, lo, hi, step=1):
    """An integer spread over the logarithm of [lo, hi], a multiple of `step`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "linear", "block", "head", "embedding", "decompress", "compress", "step"])
    step = rng.choice([64, 8, 8, 1])                    # one matrix in four has odd sizes
    tile = rng.choice([64, 128, 128, 1024])
    if kind == "linear":
        K = _size(rng, 512, 11008, step)
        N = _size(rng, 512, min(22016, 4096 * 22016 // K), step)
        M = _size(rng, 1, 16) if rng.random() < 0.6 else _size(rng, 17, min(2048, 2048 * 4096 * 22016 // (K * N)))
        return {"kind": kind, "api": rng.choice(["module", "module", "function"]) if M <= 16 else "module", "K": K, "N": N,
                "tile": tile, "M": M, "bias": rng.random() < 0.3}
    if kind == "block":
        hidden = _size(rng, 1024, 4096, 128)
        return {"kind": kind, "hidden": hidden, "ffn": _size(rng, 2 * hidden, 11008, 64), "tile": rng.choice([64, 128]),
                "M": _size(rng, 1, 16)}
    if kind == "head":
        return {"kind": kind, "V": _size(rng, 8000, 32000, step), "H": _size(rng, 1024, 4096, 64), "tile": tile,
                "M": _size(rng, 1, 8)}
    if kind == "embedding":
        return {"kind": kind, "V": _size(rng, 8000, 32000, step), "H": _size(rng, 1024, 4096, 64),
                "tile": rng.choice([16, 64, 128, 1024]), "ids": _size(rng, 1, 4096)}
    if kind in ("decompress", "compress"):
        return {"kind": kind, "K": _size(rng, 512, 11008, step), "N": _size(rng, 512, 4096, step), "tile": tile}
    hidden = _size(rng, 1024, 4096, 128)
    return {"kind": kind, "hidden": hidden, "ffn": _size(rng, 2 * hidden, 11008, 64), "vocab": _size(rng, 8000, 32000, 8),
            "layers": rng.randint(1, 2), "tile": rng.choice([64, 128]), "batch": _size(rng, 1, 8),
            "context": _size(rng, 64, 1024)}


# ------------------------------------------------------------------------------------------------ preparation

def _weight(K, N, gen):
    return (torch.randn(K, N, generator=gen, device="cuda") * 0.02).to(torch.bfloat16)


def _acts(shape, gen):
    return torch.randn(*shape, generator=gen, device="cuda").to(torch.bfloat16)


def _compressed(K, N, tile, gen):
    return ci.compress_weight_cuda(_weight(K, N, gen), tile, 32)


def _linear(K, N, tile, gen, parts=None):
    c = _compressed(K, N, tile, gen)
    th, tw = c["tile_height"], c["tile_width"]
    m = ci.RansFusedLinear(K, parts, th, tw) if parts else ci.RansLinear(K, N, th, tw)
    return m.load_compressed(c).prepare()


def _arrays(c, shape):
    """The keyword arguments that every function of the functional interface shares."""
    return dict(initial_states=c["rans_exp_states"], tables=c["rans_exp_tables"], slot_map=c["rans_exp_slot_map"],
                weight_shape=shape, tile_offsets=c["rans_exp_tile_offsets"], tile_max_lens=c["rans_exp_tile_max_lens"],
                tile_k=c["tile_height"], tile_n=c["tile_width"], mantissas=c["rans_man_raw"])


class _Norm(nn.Module):
    def __init__(self, width, gen):
        super().__init__()
        self.weight = nn.Parameter((1 + 0.1 * torch.randn(width, generator=gen, device="cuda")).to(torch.bfloat16),
                                   requires_grad=False)
        self.variance_epsilon = 1e-5


def _model(case, gen):
    """A Llama-shaped module tree on compressed projections, as patch_model leaves it with fused projections."""
    H, F, V, tile = case["hidden"], case["ffn"], case["vocab"], case["tile"]
    layers = []
    for _ in range(case["layers"]):
        q = _linear(H, 3 * H, tile, gen, [H, H, H])
        gate = _linear(H, 2 * F, tile, gen, [F, F])
        attn = SimpleNamespace(q_proj=q, k_proj=ci.RansFusedSlice(q, H, 2 * H), v_proj=ci.RansFusedSlice(q, 2 * H, 3 * H),
                               o_proj=_linear(H, H, tile, gen))
        mlp = SimpleNamespace(gate_proj=gate, up_proj=ci.RansFusedSlice(gate, F, 2 * F), down_proj=_linear(F, H, tile, gen))
        layers.append(SimpleNamespace(input_layernorm=_Norm(H, gen), post_attention_layernorm=_Norm(H, gen),
                                      self_attn=attn, mlp=mlp))
    table = _compressed(V, H, 16, gen)
    embed = ci.RansEmbedding(V, H, table["tile_height"], table["tile_width"]).load_compressed(table).prepare()
    stored = _compressed(V, H, tile, gen)
    head = ci.RansLMHead(H, V, stored["tile_height"], stored["tile_width"]).load_compressed(stored).prepare()
    config = SimpleNamespace(hidden_size=H, num_attention_heads=H // HEAD_DIM, head_dim=HEAD_DIM, rope_theta=10000.0)
    return SimpleNamespace(config=config, lm_head=head,
                           model=SimpleNamespace(embed_tokens=embed, layers=layers, norm=_Norm(H, gen)))


def prepare(case, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    kind, s = case["kind"], {"kind": case["kind"]}
    if kind == "linear":
        K, N, M = case["K"], case["N"], case["M"]
        s["x"] = _acts((M, K), gen)
        bias = _acts((N,), gen) if case["bias"] else None
        c = _compressed(K, N, case["tile"], gen)
        if case["api"] == "module":
            m = ci.RansLinear(K, N, c["tile_height"], c["tile_width"], has_bias=case["bias"])
            if bias is not None:
                m.bias = bias
            s["module"] = m.load_compressed(c).prepare()
        else:
            s["stream"], s["args"] = c["rans_exp_stream"], dict(_arrays(c, (K, N)), bias=bias)
    elif kind == "block":
        H, F, tile = case["hidden"], case["ffn"], case["tile"]
        s["x"] = [_acts((case["M"], k), gen) for k in (H, H, H, F)]
        s["linears"] = [_linear(k, n, tile, gen) for k, n in ((H, 3 * H), (H, H), (H, 2 * F), (F, H))]
    elif kind == "head":
        V, H = case["V"], case["H"]
        s["x"] = _acts((case["M"], H), gen)
        c = _compressed(V, H, case["tile"], gen)
        s["stream"], s["args"] = c["rans_exp_stream"], _arrays(c, (V, H))
    elif kind == "embedding":
        V, H = case["V"], case["H"]
        c = _compressed(V, H, case["tile"], gen)
        s["module"] = ci.RansEmbedding(V, H, c["tile_height"], c["tile_width"]).load_compressed(c).prepare()
        s["ids"] = torch.randint(0, V, (case["ids"],), generator=gen, device="cuda")
    elif kind == "decompress":
        c = _compressed(case["K"], case["N"], case["tile"], gen)
        s["stream"], s["args"] = c["rans_exp_stream"], _arrays(c, (case["K"], case["N"]))
    elif kind == "compress":
        s["weight"], s["tile"] = _weight(case["K"], case["N"], gen), case["tile"]
        s["package"] = torch.zeros(case["K"] * case["N"], dtype=torch.uint8, device="cuda")    # room for the stream
    else:
        B, ctx = case["batch"], case["context"]
        runner = LlamaGreedyRunner(_model(case, gen), B, ctx + 16)
        runner.k_cache.normal_(generator=gen)
        runner.v_cache.normal_(generator=gen)
        s["tok"] = torch.randint(0, case["vocab"], (B,), generator=gen, device="cuda")
        runner.tok.copy_(s["tok"])
        runner.pos.fill_(ctx)
        s["context"], s["runner"], s["graph"] = ctx, runner, runner.capture(B)
    return s


# ------------------------------------------------------------------------------------------------ one pass

def run(s):
    kind = s["kind"]
    if kind in ("linear", "embedding") and "module" in s:
        return s["module"](s["x"] if kind == "linear" else s["ids"])
    if kind == "linear":
        return ci.fused_rans_linear_triton(s["x"], s["stream"], **s["args"])
    if kind == "block":
        return [m(x) for m, x in zip(s["linears"], s["x"])]
    if kind == "head":
        return ci.fused_rans_linear_transposed_triton(s["x"], s["stream"], **s["args"])
    if kind == "decompress":
        return ci.rans_decompress_bf16(s["stream"], **s["args"])
    if kind == "compress":
        c = ci.compress_weight_cuda(s["weight"], s["tile"], 32)
        stream = c["rans_exp_stream"]                   # its length depends on the weight: it goes into a package of fixed size
        s["package"][:stream.numel()].copy_(stream)
        return [s["package"], stream.numel()] + [c[k] for k in (
            "rans_exp_states", "rans_exp_tables", "rans_exp_slot_map", "rans_man_raw", "rans_exp_tile_offsets",
            "rans_exp_tile_max_lens", "output_sizes", "exponent_freqs", "exponent_cdf")]
    r = s["runner"]                                     # one serving step at the same position again
    r.tok.copy_(s["tok"])
    r.pos.fill_(s["context"])
    r.steps_done.zero_()
    s["graph"].replay()
    return [r.logits, r.k_cache, r.v_cache]


# ------------------------------------------------------------------------------------------------ bounds

def _packed(K, N, tile):
    """Bytes of a compressed [K, N] weight: sign+mantissa plane, exponent stream at the entropy of N(0, s) plus its
    12-bit table's loss, one state per stream."""
    while tile > K and tile > 1:
        tile //= 2
    return K * N * (1 + 2.64 / 8) + -(-K // tile) * 2 * N * 4


def work(case):
    kind = case["kind"]
    if kind == "linear":
        K, N, M = case["K"], case["N"], case["M"]
        return {"bytes": _packed(K, N, case["tile"]) + 2 * M * (K + N), "flops": 2 * M * K * N}
    if kind == "block":
        H, F, M = case["hidden"], case["ffn"], case["M"]
        mats = ((H, 3 * H), (H, H), (H, 2 * F), (F, H))
        return {"bytes": sum(_packed(k, n, case["tile"]) + 2 * M * (k + n) for k, n in mats),
                "flops": sum(2 * M * k * n for k, n in mats)}
    if kind == "head":
        V, H, M = case["V"], case["H"], case["M"]
        return {"bytes": _packed(V, H, case["tile"]) + 2 * M * (V + H), "flops": 2 * M * V * H}
    if kind == "embedding":
        return {"bytes": case["ids"] * (case["H"] * (2 + 1 + 2.64 / 8) + 8), "flops": 0}
    if kind in ("decompress", "compress"):
        K, N = case["K"], case["N"]
        return {"bytes": 2 * K * N + _packed(K, N, case["tile"]), "flops": 0}
    H, F, V, L, B, ctx = (case[k] for k in ("hidden", "ffn", "vocab", "layers", "batch", "context"))
    mats = [(H, 3 * H), (H, H), (H, 2 * F), (F, H)] * L + [(H, V)]
    return {"bytes": sum(_packed(k, n, case["tile"]) + 2 * B * (k + n) for k, n in mats) + 4 * L * B * ctx * H,
            "flops": sum(2 * B * k * n for k, n in mats) + 4 * L * B * ctx * H}


def tolerance(case):
    if case["kind"] in ("embedding", "decompress", "compress"):
        return "exact"
    return {"rel": 1e-2, "max": 0.1}
