"""The work that is timed: what a program built on flint_b200 has the GPU do, through the public entry points.

Five kinds of pass, in the proportions of a chat or speculative-decoding program:

  decode   one token of a batch-1 stream, chained on the device as `generate` does it (`DecodeEngine.decode_chained`)
  verify   M candidate tokens scored in one weight pass (`DecodeEngine.verify`): a token tree with its mask, or a chain
           called as `generate(draft_model=...)` calls it, without mask or depths
  prefill  a prompt through the model facade (`Transformer.forward` with `return_hidden`, the first step of `generate`)
  draft    the EAGLE draft head: one forward over T rows (the context window, a beam level, a single rollout step), then
           the token head
  sample   token choice from a logits buffer (`DecodeEngine.sample`)

The shapes are the repository's own model configurations; weights are seeded normal matrices quantised by the library's
packers. The projections that write the residual stream (O, down) are scaled by 1 / sqrt(2 * layers), the usual
initialisation of a deep pre-norm decoder, and the embeddings of models without an embedding multiplier have about unit
variance: the stream then grows slowly with depth, as it does in trained models.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import torch

from flint_b200 import packing
from flint_b200.config import ModelArgs
from flint_b200.draft import DraftHead
from flint_b200.engine import DecodeEngine
from flint_b200.model import Transformer
from flint_b200.tree import static_tree, tree_mask

DEV = "cuda"


def listed():
    return [
        # chat at a temperature: the token is drawn from the last step's logits, large vocabulary
        dict(name="sample-topk", kind="sample", rows=1, vocab=128256, temperature=0.8, top_k=50),
        # one step of a draft rollout: a single row, then its token; the smallest weight-bound call
        dict(name="draft-step", kind="draft", model="granite-3b-class", rows=1, window=32, heads=1, top_b=1),
        # the context window that primes a rollout
        dict(name="draft-window", kind="draft", model="granite-3b-class", rows=32, window=32, heads=1, top_b=1),
        # the first tokens of an answer of the smallest model: latency only
        dict(name="decode-1b-start", kind="decode", model="llama-1b-class", pos=21, asym=False),
        # the headline: a short chat with the 3B-class model
        dict(name="decode-3b", kind="decode", model="granite-3b-class", pos=200, asym=False),
        # the model shape that the reference's own kernels run (40 / 8 heads of 64, scalar multipliers), a few turns in
        dict(name="decode-ref-shape", kind="decode", model="granite-4.1-3b", pos=603, asym=False),
        # the largest model with gpt-fast's asymmetric weights, in the middle of a document
        dict(name="decode-8b-asym", kind="decode", model="llama-8b-class", pos=1777, asym=True),
        # long context: as many bytes of K / V as of weights, twice over
        dict(name="decode-3b-32k", kind="decode", model="granite-3b-class-32k", pos=32768, asym=False),
        # chain speculation with K = 3: four candidates
        dict(name="verify-3b-chain4", kind="verify", model="granite-3b-class", m=4, tree=False, pos=301, asym=False),
        # the static 26-node tree over 1024 cached positions
        dict(name="verify-3b-tree26", kind="verify", model="granite-3b-class", m=26, tree=True, pos=1024, asym=False),
        # the widest tree on the largest model, late in a conversation
        dict(name="verify-8b-tree61", kind="verify", model="llama-8b-class", m=61, tree=True, pos=3001, asym=False),
        # a prompt of ordinary length, not a multiple of anything
        dict(name="prefill-3b", kind="prefill", model="granite-3b-class", tokens=725, asym=False),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choices(("decode", "verify", "prefill", "draft", "sample"), (7, 5, 3, 3, 2))[0]
    if kind == "sample":
        temperature = rng.choice((0.0, 0.6, 0.8, 1.0))
        return dict(kind=kind, rows=_log(rng, 1, 64), vocab=rng.choice((49160, 100352, 128256)), temperature=temperature,
                    top_k=rng.choice((0, 10, 50, 200)) if temperature else 0)
    if kind == "draft":
        window = rng.choice((16, 32, 48))
        rows = rng.choice((1, rng.randint(2, window), window))
        return dict(kind=kind, model=rng.choice(("granite-3b-class", "granite-4.1-3b", "llama-1b-class")), rows=rows,
                    window=window, heads=rng.choice((1, 2, 4)), top_b=rng.choice((1, 2, 4)))
    asym = rng.random() < 0.2
    if kind == "prefill":
        model = rng.choice(("llama-1b-class", "granite-3b-class", "granite-4.1-3b", "llama-8b-class"))
        return dict(kind=kind, model=model, tokens=_log(rng, 17, 290 if "8b" in model else 680), asym=asym)
    model = rng.choice(("llama-1b-class", "granite-3b-class", "granite-4.1-3b", "llama-8b-class", "granite-3b-class-32k"))
    if kind == "decode":
        return dict(kind=kind, model=model, pos=_log(rng, 1, 32768 if "32k" in model else 4000), asym=asym)
    return dict(kind=kind, model=model, m=_log(rng, 2, 64), tree=rng.random() < 0.6, pos=_log(rng, 16, 4000), asym=asym)


def _weights(cfg, seed, asym):
    packed = packing.synth_packed(cfg, seed, device=DEV, asym=asym)
    for n in ("o_s", "d_s", "o_z", "d_z"):
        if n in packed:
            packed[n] *= (2 * cfg.n_layer) ** -0.5
    if cfg.embedding_multiplier == 1.0:
        packed["embed"] *= 64.0
    return packed


def _fill(cache, pos, gen):
    for layer in cache:                      # per layer: one stacked fp32 intermediate would be twice the cache
        layer[:pos].normal_(generator=gen)


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    kind = case["kind"]
    s = SimpleNamespace(case=case, kind=kind)
    if kind == "sample":
        s.engine = _sampler()
        s.logits = torch.randn(case["rows"], case["vocab"], generator=gen, device=DEV) * 2.5
        s.seed = seed
        return s
    cfg = ModelArgs.from_name(case["model"])
    if kind == "draft":
        head = DraftHead(cfg.dim, cfg.n_head, cfg.intermediate_size, rope_base=cfg.rope_base)
        head.load_state_dict({k: torch.randn(shp, generator=gen, device=DEV) * 0.02 if len(shp) == 2 else torch.ones(shp, device=DEV)
                              for k, shp in head.state_shapes().items()}, device=DEV)
        embed = (torch.randn(cfg.vocab_size, cfg.dim, generator=gen, device=DEV) * 0.02).to(torch.bfloat16)
        head.bind_target(embed, torch.ones(cfg.dim, dtype=torch.bfloat16, device=DEV), cfg.logits_scaling)
        window, rows = case["window"], case["rows"]
        head.setup_cache(window + 8)
        feat = torch.randn(window, cfg.dim, generator=gen, device=DEV).to(torch.bfloat16)
        tokens = torch.randint(0, cfg.vocab_size, (window,), generator=gen, device=DEV, dtype=torch.int32)
        slots = torch.arange(window, dtype=torch.int32, device=DEV)
        if rows == window:                   # the window itself
            s.feat, s.tokens, s.slots = feat, tokens, slots
        else:                                # later rows, behind a window that is in the cache already
            head(feat, None, slots, input_pos=slots, tokens=tokens)
            first = min(window, window + 8 - rows)      # more rows than free slots replace the window's last ones
            s.feat, s.tokens = feat[:rows].contiguous(), tokens[:rows].contiguous()
            s.slots = torch.arange(first, first + rows, dtype=torch.int32, device=DEV)
        s.rows = torch.randn(case["heads"], cfg.dim, generator=gen, device=DEV).to(torch.bfloat16)
        s.head = head
        return s
    packed = _weights(cfg, seed, case["asym"])
    if kind == "prefill":
        s.model = Transformer(cfg).load_packed(packed)
        s.model.setup_caches(1, case["tokens"] + 64)
        s.idx = torch.randint(0, cfg.vocab_size, (1, case["tokens"]), generator=torch.Generator().manual_seed(seed))
        s.input_pos = torch.arange(case["tokens"])
        eng = s.model.engine
        s.rows = (eng.kc[:, :case["tokens"]], eng.vc[:, :case["tokens"]])
        return s
    pos, m = case["pos"], case.get("m", 1)
    eng = DecodeEngine(cfg, packed, max_seq=(pos + m + 255) // 256 * 256)
    _fill(eng.kc, pos, gen)
    _fill(eng.vc, pos, gen)
    s.engine, s.pos = eng, pos
    s.rows = (eng.kc[:, pos:pos + m], eng.vc[:, pos:pos + m])
    s.tokens = torch.randint(0, cfg.vocab_size, (m,), generator=gen, device=DEV, dtype=torch.int32)
    if kind == "decode":
        s.next = torch.zeros(1, dtype=torch.int32, device=DEV)
        s.logits = torch.empty(cfg.vocab_size, dtype=torch.float32, device=DEV)
    elif case["tree"]:
        parent, depth = static_tree(m)
        s.depth = torch.tensor(depth, dtype=torch.int32, device=DEV)
        s.amask = torch.from_numpy(tree_mask(parent)).to(DEV)
    return s


_tiny = []


def _sampler():
    """Any engine samples from any logits buffer: the smallest model stands in for the one that wrote it."""
    if not _tiny:
        cfg = ModelArgs.from_name("tiny")
        _tiny.append(DecodeEngine(cfg, packing.synth_packed(cfg, 0, device=DEV), max_seq=32))
    return _tiny[0]


def run(s):
    c = s.case
    if s.kind == "sample":
        return s.engine.sample(s.logits, c["temperature"], c["top_k"] or None, seed=s.seed, counter=7)
    if s.kind == "draft":
        out = s.head(s.feat, None, s.slots, input_pos=s.slots, tokens=s.tokens)
        tokens, scores = s.head.head(s.rows, top_b=c["top_b"], want_scores=True)
        return out, tokens, scores
    if s.kind == "prefill":
        logits, hidden = s.model(s.idx, s.input_pos, return_hidden=True)
        return logits, hidden, s.rows
    if s.kind == "decode":
        # the arg-max token is a function of the logits, and of the order of a sum where two logits nearly tie
        s.engine.decode_chained(s.tokens, s.pos, s.next, s.logits)
        return s.logits, s.rows
    if c["tree"]:
        logits, feat = s.engine.verify(s.tokens, s.pos, s.depth, s.amask)
    else:
        logits, feat = s.engine.verify(s.tokens, s.pos)
    return logits, feat, s.rows


def work(case):
    kind = case["kind"]
    if kind == "sample":
        return {"bytes": 4 * case["rows"] * (case["vocab"] + 1), "flops": 0}
    cfg = ModelArgs.from_name(case["model"])
    d = cfg.dim
    if kind == "draft":
        block = 2 * d * d + 4 * d * d + 3 * d * cfg.intermediate_size + d * d
        rows, heads = case["rows"], case["heads"]
        kv = 2 * 2 * d * (case["window"] + 8)
        return {"bytes": 2 * (block + cfg.vocab_size * d) + 2 * d * (3 * rows + heads) + kv + 8 * heads * case["top_b"],
                "flops": 2 * (block * rows + cfg.vocab_size * d * heads)}
    m = case["tokens"] if kind == "prefill" else case.get("m", 1)
    pos = 0 if kind == "prefill" else case["pos"]
    kv_row = 2 * 2 * cfg.n_layer * cfg.n_local_heads * cfg.head_dim
    out = m * (4 * cfg.vocab_size + kv_row + 2 * d + (2 * d if kind != "decode" else 0))
    seen = m * pos + m * (m + 1) // 2
    return {"bytes": cfg.bytes_per_token(pos, case["asym"]) + out,
            "flops": 2 * m * cfg.int4_params() + 4 * seen * cfg.n_layer * cfg.n_head * cfg.head_dim}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case["kind"] == "draft":                    # one layer, every sub-result rounded to bf16
        return {"rel": 0.01}
    # 16 to 40 layers whose residual stream and branch results are rounded to bf16 (2^-9) six times each: where two
    # implementations sum in another order a rounding flips here and there and the flips spread. The GEMM implementations
    # that the library has side by side differ by 1.0e-2 to 1.7e-2 on these models (largest value 0.1).
    return {"rel": 0.025, "max": 0.25}
