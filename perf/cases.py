"""The work that users of glorcq_b200 have it do, as cases that can be timed and compared.

Five kinds, each through the entry point a program calls:

  linear   one GLoRCQLinear on a batch of rows: 2-/4-bit integer codes, 3-bit codes (the int8 kernel), codebook codes
           behind a rotation
  grouped  turbo_dequant_grouped_gemv_fused, the row-major drop-in a host with its own MoE loop calls
  moe      one GraphCompatibleMoeBlock, called eagerly
  decode   one token per sequence of a decoder through GLoRCQGraphWrapper.replay
  prefill  the prompt pass of a decoder, the logits of the last position kept

Weights and activations are drawn as in the benchmark: uniform codes, scales |N(0, 0.02)|, integer zero points, low-rank
factors N(0, 0.01), activations N(0, 1), uniformly drawn token ids."""

import math
from types import SimpleNamespace

import torch

from glorcq_b200 import tiled
from glorcq_b200.graph_wrapper import GLoRCQGraphWrapper, StaticCache
from glorcq_b200.hadamard_rotation import generate_rht_signs
from glorcq_b200.kernels import turbo_dequant_grouped_gemv_fused
from glorcq_b200.model_builder import RotationCache
from glorcq_b200.moe_block import GraphCompatibleMoeBlock
from glorcq_b200.quantized_linear import GLoRCQLinear
from glorcq_b200.synthetic import MIXTRAL_8X7B, QWEN15_MOE_A27B, QWEN3_30B_A3B, make_decoder

MODELS = {"qwen15": QWEN15_MOE_A27B, "mixtral": MIXTRAL_8X7B, "qwen3": QWEN3_30B_A3B}
BITS = {"q2": 2, "q3": 3, "q4": 4, "t2": 2}
GROUP = 128
SYMMETRIC_CODEBOOK = (-1.510, -0.4528, 0.4528, 1.510)     # the four levels of a unit normal's best 2-bit quantizer


def listed():
    return [
        # the smallest call: one expert projection on one token
        {"name": "linear-q2-1", "kind": "linear", "fmt": "q2", "rows": 1, "N": 1408, "K": 2048, "rank": 64, "rotation": "none"},
        # an attention projection on a ragged prompt
        {"name": "linear-q4-333", "kind": "linear", "fmt": "q4", "rows": 333, "N": 4096, "K": 4096, "rank": 64, "rotation": "none"},
        # codebook weights see rotated activations: a small decode batch through rotation, low-rank term and product
        {"name": "linear-codebook-5", "kind": "linear", "fmt": "t2", "rows": 5, "N": 5632, "K": 2048, "rank": 64, "rotation": "hadamard"},
        # code widths that are not re-tiled
        {"name": "linear-3bit-2", "kind": "linear", "fmt": "q3", "rows": 2, "N": 2048, "K": 2048, "rank": 64, "rotation": "none"},
        # the four experts of one token, row-major operands
        {"name": "grouped-codebook-4", "kind": "grouped", "E": 4, "N": 1408, "K": 2048},
        # one decoder block's experts for a token, for a decode batch, and in the codebook format for an odd batch
        {"name": "moe-qwen15-1", "kind": "moe", "model": "qwen15", "fmt": "q2", "tokens": 1, "rank": 64},
        {"name": "moe-qwen15-32", "kind": "moe", "model": "qwen15", "fmt": "q2", "tokens": 32, "rank": 64},
        {"name": "moe-qwen15-codebook-9", "kind": "moe", "model": "qwen15", "fmt": "t2", "tokens": 9, "rank": 64},
        # the headline: one token of the whole model after a 512-token prompt; and that prompt itself
        {"name": "decode-qwen15-1", "kind": "decode", "model": "qwen15", "layers": 24, "batch": 1, "context": 512},
        {"name": "prefill-qwen15-512", "kind": "prefill", "model": "qwen15", "layers": 24, "batch": 1, "tokens": 512},
        # batched decode of wide experts after a 1024-token prompt (the layers repeat: four of the 32)
        {"name": "decode-mixtral-16", "kind": "decode", "model": "mixtral", "layers": 4, "batch": 16, "context": 1024},
        # a long prompt over many small experts (six of the 48 layers)
        {"name": "prefill-qwen3-4096", "kind": "prefill", "model": "qwen3", "layers": 6, "batch": 1, "tokens": 4096},
    ]


def _spread(rng, lo, hi, step=1):
    """A multiple of `step` from lo to hi, even over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))
    return min(hi, max(lo, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(("linear", "linear", "grouped", "moe", "moe", "decode", "prefill"))
    if kind == "linear":
        fmt = rng.choice(("q2", "q2", "q4", "t2", "q3"))
        return {"kind": kind, "fmt": fmt, "rows": _spread(rng, 1, 32 if fmt == "q3" else 2048), "N": _spread(rng, 512, 14336, 8),
                "K": _spread(rng, 768, 5632, 128), "rank": rng.choice((0, 32, 64, 128)),
                "rotation": rng.choice(("hadamard", "qr")) if fmt == "t2" else "none"}
    if kind == "grouped":
        return {"kind": kind, "E": _spread(rng, 1, 64), "N": _spread(rng, 512, 4096, 8), "K": _spread(rng, 768, 4096, 128)}
    if kind == "moe":
        return {"kind": kind, "model": rng.choice(("qwen15", "mixtral", "qwen3")), "fmt": rng.choice(("q2", "q2", "q4", "t2")),
                "tokens": _spread(rng, 1, 2048), "rank": rng.choice((32, 64, 128))}
    model = rng.choice(("qwen15", "mixtral", "qwen3"))
    if kind == "decode":
        return {"kind": kind, "model": model, "layers": rng.randint(1, 4), "batch": _spread(rng, 1, 16 if model == "mixtral" else 64),
                "context": _spread(rng, 16, 1024)}
    return {"kind": kind, "model": model, "layers": rng.randint(1, 4), "batch": 1, "tokens": _spread(rng, 16, 4096)}


# ---- weights --------------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _normal(g, *shape, scale=1.0):
    return (torch.randn(*shape, generator=g, device="cuda") * scale).half()


def _rotation(g, K, rotation):
    """The codebook format's rotation: a cache with the codebook and an orthogonal matrix, and the signs of the Hadamard form."""
    cache = RotationCache(device="cuda")
    if rotation == "qr":
        Pi = torch.linalg.qr(torch.randn(K, K, generator=g, device="cuda"))[0]
    else:
        Pi = torch.zeros(1, 1)
    cache.put(K, 2, 42, Pi, torch.tensor(SYMMETRIC_CODEBOOK) / math.sqrt(K))
    return cache, generate_rht_signs(K) if rotation == "hadamard" else None


def _linear(g, N, K, fmt, rank, U=None, rot=None):
    lin = GLoRCQLinear(K, N)
    if fmt == "t2":
        lin.load_turbo({"packed_indices": torch.randint(0, 256, (N, K // 4), generator=g, device="cuda", dtype=torch.uint8),
                        "norms": torch.rand(N, generator=g, device="cuda") + 0.5, "bits": 2, "dim": K, "seed": 42}, rot[0])
        lin._rht_signs = rot[1]
    else:
        groups, bits = -(-K // GROUP), BITS[fmt]
        lin.load_gptq({"qweight_int": torch.randint(0, 2 ** bits, (N, K), generator=g, device="cuda", dtype=torch.int32),
                       "scales": _normal(g, N, groups, scale=0.02).abs(),
                       "zeros": torch.randint(0, 2 ** bits, (N, groups), generator=g, device="cuda").half(),
                       "bits": bits, "groupsize": GROUP, "sym": False}, check_range=False)
    if rank:
        lin.load_sv(_normal(g, K, rank, scale=0.01) if U is None else U, _normal(g, N, rank, scale=0.01))
    return lin


def _sizes(model):
    """hidden, expert width, experts, experts of a token, shared expert's width"""
    m = MODELS[model]
    return (m["hidden_size"], m.get("moe_intermediate_size") or m["intermediate_size"], m.get("num_experts") or m["num_local_experts"],
            m["num_experts_per_tok"], m.get("shared_expert_intermediate_size", 0))


def _moe_block(g, model, fmt, rank):
    H, I, E, k, Ish = _sizes(model)
    rot = {K: _rotation(g, K, "hadamard") for K in {H, I, Ish} if K} if fmt == "t2" else {}
    pools = {}

    def expert(width, cluster):
        def proj(name, N, K):
            if (name, cluster) not in pools:        # U is shared by the experts of a cluster
                pools[name, cluster] = _normal(g, K, rank, scale=0.01)
            return _linear(g, N, K, fmt, rank, pools[name, cluster], rot.get(K))
        return SimpleNamespace(gate_proj=proj("gate", width, H), up_proj=proj("up", width, H), down_proj=proj("down", H, width))

    def dense(rows):
        lin = torch.nn.Linear(H, rows, bias=False, device="cuda", dtype=torch.float16)
        lin.weight.data.copy_(_normal(g, rows, H, scale=0.02))
        return lin

    block = SimpleNamespace(num_experts=E, top_k=k, norm_topk_prob=MODELS[model].get("norm_topk_prob", model == "mixtral"), gate=dense(E),
                            experts=[expert(I, e // 4) for e in range(E)], shared_expert=expert(Ish, "shared") if Ish else None,
                            shared_expert_gate=dense(1) if Ish else None)
    return GraphCompatibleMoeBlock(block).prepare("cuda", release_linear_tiles=True)


_model = (None, None)


def _decoder(model, layers):
    """A program loads its model once and serves every request with it: the last one is kept."""
    global _model
    if _model[0] != (model, layers):
        _model = (None, None)
        tiled.clear_pool()
        torch.cuda.empty_cache()
        _model = ((model, layers), make_decoder(dict(MODELS[model], num_hidden_layers=layers), "cuda:0").eval())
    return _model[1]


# ---- one pass -------------------------------------------------------------------------------------
def prepare(case, seed):
    g, kind = _generator(seed), case["kind"]
    if kind == "linear":
        rot = _rotation(g, case["K"], case["rotation"]) if case["fmt"] == "t2" else None
        lin = _linear(g, case["N"], case["K"], case["fmt"], case["rank"], rot=rot)
        return {"kind": kind, "layer": lin, "x": _normal(g, case["rows"], case["K"])}
    if kind == "grouped":
        E, N, K = case["E"], case["N"], case["K"]
        return {"kind": kind, "N": N, "x": _normal(g, E, K),
                "packed": torch.randint(0, 256, (E * N, K // 4), generator=g, device="cuda", dtype=torch.uint8),
                "norms": torch.rand(E * N, generator=g, device="cuda") + 0.5,
                "codebook": torch.tensor(SYMMETRIC_CODEBOOK, device="cuda") / math.sqrt(K)}
    if kind == "moe":
        block = _moe_block(g, case["model"], case["fmt"], case["rank"])
        return {"kind": kind, "block": block, "x": _normal(g, 1, case["tokens"], _sizes(case["model"])[0])}
    model = _decoder(case["model"], case["layers"])
    B, T = case["batch"], case.get("context") or case["tokens"]
    ids = torch.randint(0, model.config.vocab_size, (B, T), generator=g, device="cuda")
    positions = torch.arange(T, device="cuda")
    if kind == "prefill":
        cache = StaticCache(model.config, B, T, torch.device("cuda:0"))
        return {"kind": kind, "model": model, "ids": ids, "positions": positions, "cache": cache}
    wrapper = GLoRCQGraphWrapper(model, max_batch_size=B, max_seq_len=T + 1)
    wrapper.capture_graph()
    wrapper.static_cache.reset()
    with torch.no_grad():
        model(input_ids=ids, cache_position=positions, past_key_values=wrapper.static_cache, logits_to_keep=1)
    kv = wrapper.static_cache.k[:, :, :, T], wrapper.static_cache.v[:, :, :, T]
    return {"kind": kind, "wrapper": wrapper, "position": T, "written": kv,
            "ids": torch.randint(0, model.config.vocab_size, (B, 1), generator=g, device="cuda")}


@torch.no_grad()
def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["layer"](state["x"])
    if kind == "grouped":
        return turbo_dequant_grouped_gemv_fused(state["x"], state["packed"], state["norms"], state["codebook"], state["N"])
    if kind == "moe":
        return state["block"](state["x"])
    if kind == "decode":
        return state["wrapper"].replay(state["ids"], state["position"]), state["written"]
    cache = state["cache"]
    logits = state["model"](input_ids=state["ids"], cache_position=state["positions"], past_key_values=cache, logits_to_keep=1)[0]
    return logits, cache.k, cache.v


# ---- what a pass cannot do without ----------------------------------------------------------------
def _linear_work(N, K, fmt, rank, rows, loads=1.0):
    """Bytes and operations of `rows` rows through one projection whose weights are read `loads` times (the share of experts hit)."""
    weights = N * K * BITS[fmt] / 8 + (4 * N if fmt == "t2" else 4 * N * -(-K // GROUP)) + 2 * rank * (N + K)
    return loads * weights + 2 * rows * (N + K), 2 * rows * (N * K + rank * (N + K))


def _moe_work(model, fmt, rank, shared_rank, tokens):
    H, I, E, k, Ish = _sizes(model)
    hit = E * (1 - (1 - k / E) ** tokens)
    parts = [_linear_work(I, H, fmt, rank, 0, 2 * hit), _linear_work(H, I, fmt, rank, 0, hit)]
    flops = 2 * tokens * k * (3 * H * I + 3 * rank * (H + I)) + 2 * tokens * E * H
    if Ish:
        parts += [_linear_work(Ish, H, fmt, shared_rank, 0, 2), _linear_work(H, Ish, fmt, shared_rank, 0)]
        flops += 2 * tokens * (3 * H * Ish + 3 * shared_rank * (H + Ish))
    return sum(p[0] for p in parts) + 2 * E * H + 2 * tokens * (2 * H + E), flops


def work(case):
    kind = case["kind"]
    if kind == "linear":
        b, f = _linear_work(case["N"], case["K"], case["fmt"], case["rank"], case["rows"])
        return {"bytes": b, "flops": f}
    if kind == "grouped":
        E, N, K = case["E"], case["N"], case["K"]
        return {"bytes": E * (N * K / 4 + 4 * N + 2 * K + 2 * N), "flops": 2 * E * N * K}
    if kind == "moe":
        b, f = _moe_work(case["model"], case["fmt"], case["rank"], case["rank"], case["tokens"])
        return {"bytes": b, "flops": f}
    m = MODELS[case["model"]]
    H, V, B, new = m["hidden_size"], m["vocab_size"], case["batch"], case.get("tokens", 1)
    heads, kv = m["num_attention_heads"], m["num_key_value_heads"]
    D, seen = m.get("head_dim", H // heads), case.get("context", 0)
    rows = B * new
    parts = [_linear_work(N, K, "q4", 64, 0) for N, K in ((heads * D, H), (kv * D, H), (kv * D, H), (H, heads * D))]
    flops = sum(_linear_work(N, K, "q4", 64, rows)[1] for N, K in ((heads * D, H), (kv * D, H), (kv * D, H), (H, heads * D)))
    flops += 4 * B * heads * D * (new * seen + new * (new + 1) / 2)
    moe = _moe_work(case["model"], "q2", 64, 0, rows)
    per_layer = sum(p[0] for p in parts) + moe[0] + 2 * 2 * B * kv * D * (seen + new)
    return {"bytes": case["layers"] * per_layer + 2 * V * H + 2 * B * V + 2 * H * rows,
            "flops": case["layers"] * (flops + moe[1]) + 2 * B * V * H}


def tolerance(case):
    """16-bit results of fp32 sums.  Where a router decides, a rounding may send a token to another expert: one token's row then
    differs by that expert's share, and in a decoder so does what follows from it."""
    if case["kind"] in ("linear", "grouped"):
        return {"rel": 1e-3}
    return {"rel": 2e-3 if case["kind"] == "moe" else 2e-2, "max": 0.9}
