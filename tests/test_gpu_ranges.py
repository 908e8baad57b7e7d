"""GPU: the ends of the ranges that the kernels' dispatch rules cut: chunks and ring stages of the decode attention, token tiles of the
verify GEMMs and the prompt pass, weight scales too far apart for the short dequantisation, row slices of the token choice,
row tiles of the draft head. Against the CPU oracle (or, for the token choice, the exact order of the input)."""
import ctypes

import geometry
import numpy as np
import pytest
import torch

from flint_b200 import _lib, packing
from flint_b200.config import ModelArgs
from flint_b200.draft import seeded_draft
from flint_b200.engine import DecodeEngine, query
from flint_b200.tree import tree_mask
from oracle import oracle as O
from oracle.draft_oracle import DraftOracle, sample_probs

pytestmark = pytest.mark.gpu


def _tol(ref):
    """2e-2 at the tiny config's largest |logit| of 2.56, the same relative bar elsewhere: the oracle alone moves by this much
    when one bf16 ulp of one input element is flipped (tests/test_packer_oracle.py)."""
    return 2e-2 * max(1.0, float(np.abs(ref).max()) / 2.56)


def _f32(t):
    return O.bf16_to_f32(t.detach().cpu().contiguous().view(torch.int16).numpy().view(np.uint16))


def _pair(cfg, max_seq, T0, P=None, seed=7):
    """Oracle and engine with the same T0 random cache rows; every later row of the device cache is NaN."""
    P = packing.synth_packed(cfg, 0) if P is None else P
    orc = O.OracleModel(cfg, P, max_seq)
    eng = DecodeEngine(cfg, {k: v.cuda() for k, v in P.items()}, max_seq=max_seq)
    kv = torch.randn(2, cfg.n_layer, T0, cfg.n_local_heads, cfg.head_dim, generator=torch.Generator().manual_seed(seed)).bfloat16()
    eng.kc.fill_(float("nan"))
    eng.vc.fill_(float("nan"))
    for cache, host, rows in ((eng.kc, orc.kc, kv[0]), (eng.vc, orc.vc, kv[1])):
        cache[:, :T0].copy_(rows)
        host[:, :T0] = rows.view(torch.int16).numpy().view(np.uint16)
    return orc, eng


def test_a_refused_cache_leaves_the_bound_one_in_place():
    """fb_bind_kv of a cache that no tensor map can describe (4 layers of 2^31 - 1 positions: more than 2^32 rows) is an error, and the next
    step runs on the cache that was bound before."""
    cfg = ModelArgs.from_name("tiny")
    orc, eng = _pair(cfg, 16, 5)
    k, v = (torch.zeros_like(eng.kc) for _ in range(2))
    rc = eng.lib.fb_bind_kv(eng._ctx, ctypes.c_void_p(k.data_ptr()), ctypes.c_void_p(v.data_ptr()), 2 ** 31 - 1)
    assert rc == _lib.FB_ERR_CUDA
    ref = orc.decode(17, 5)
    with pytest.raises(_lib.FlintError):
        eng.decode(17, 16)                                    # still the bound cache's length
    got = eng.decode(17, 5).cpu().numpy()
    eng.check()
    assert np.abs(got - ref).max() < _tol(ref) and not k.any() and not v.any()
    eng.close()


# (head_dim, query heads per kv head, positions per ring stage)
SHAPES = {"llama-1b-class": 64, "granite-4.1-3b": 64, "granite-3b-class": 64, "llama-8b-class": 32}


@pytest.mark.parametrize("T0", ["one", "unit", "stage-1", "stage", "chunk-1", "chunk", "chunk+1", "many"])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_decode_attention_at_unit_stage_and_chunk_edges(name, T0):
    """Cached lengths where this step's own row is the only one, starts a unit of 16, ends or opens a ring stage, a chunk (two stages) or a
    second chunk, for every head geometry; one layer, 512 tokens of vocabulary."""
    nps = SHAPES[name]
    pos = {"one": 0, "unit": 16, "stage-1": nps - 1, "stage": nps, "chunk-1": 2 * nps - 1, "chunk": 2 * nps, "chunk+1": 2 * nps + 1,
           "many": 39 * nps + 5}[T0]
    cfg = ModelArgs.from_name(name)
    cfg.n_layer, cfg.vocab_size = 1, 512
    orc, eng = _pair(cfg, pos + 4, pos)
    for i, t in enumerate((17, 400)):
        ref = orc.decode(t, pos + i)
        got = eng.decode(t, pos + i).cpu().numpy()
        eng.check()
        assert np.abs(got - ref).max() < _tol(ref)
    eng.close()


@pytest.mark.parametrize("name", sorted(SHAPES))
def test_decode_stages_that_warps_wrote_to_are_handed_back_whole(name):
    """The attention stores this step's own row and zeros into ring stages that the weight stream takes over next: 100 launches at ragged
    lengths (several units and stages per chunk) give the same bits every time, and the first of them the oracle's values."""
    cfg = ModelArgs.from_name(name)
    cfg.n_layer, cfg.vocab_size = 2, 512
    for pos in (SHAPES[name] + 3, 21 * SHAPES[name] + 9):
        orc, eng = _pair(cfg, pos + 4, pos)
        ref, first = orc.decode(17, pos), eng.decode(17, pos).clone()
        assert np.abs(first.cpu().numpy() - ref).max() < _tol(ref)
        other = torch.zeros((), dtype=torch.int64, device="cuda")
        for _ in range(100):
            other += (eng.decode(17, pos) != first).sum()
        eng.check()
        assert int(other) == 0
        eng.close()


@pytest.mark.parametrize("asym", [False, True])
@pytest.mark.parametrize("M", [17, 32, 33, 63, 64])
def test_verify_token_tile_edges(M, asym):
    """The token tiles of the tree GEMMs and the row tiles of the attention: one past and exactly full tiles, the largest tree."""
    cfg = ModelArgs.from_name("tiny")
    orc, eng = _pair(cfg, 128, 9, packing.synth_packed(cfg, 0, asym=asym))
    toks = torch.randint(0, cfg.vocab_size, (M,), generator=torch.Generator().manual_seed(M)).tolist()
    ref, _ = orc.verify(toks, 9)
    lg, _ = eng.verify(toks, 9)
    eng.check()
    assert np.abs(lg.cpu().numpy() - ref).max() < _tol(ref)
    assert np.abs(_f32(eng.kc[:, 9:9 + M]) - O.bf16_to_f32(orc.kc[:, 9:9 + M])).max() < 0.05
    eng.close()


@pytest.mark.parametrize("asym", [False, True])
@pytest.mark.parametrize("name,M,pos", [("tiny", 1, 0), ("tiny", 3, 0), ("tiny", 40, 0), ("tiny", 70, 0), ("tiny", 300, 0), ("tiny", 3, 600),
                                        ("tiny", 16, 600), ("llama-1b-class", 26, 1000), ("llama-1b-class", 70, 0)])
def test_passes_that_give_up_leave_nothing_behind(name, M, pos, asym):
    """With a wait limit of 0 a pass (one token: a decode step; up to 64 a tree pass; more a prompt pass) gives up at the first wait that is not
    satisfied already. Every launch ends, after its copies, MMAs and remote stores in flight (their wait has its own limit), the status says
    time-out or, if every wait happened to be satisfied, nothing, and the next clean pass gives the bits of the first. Behind 600 positions the
    attention of 3 and 16 tokens runs as clusters of eight whose partials are asynchronous stores, at position 0 as one CTA; the larger model's
    prompt runs as clusters of four that share K."""
    cfg = ModelArgs.from_name(name)
    if name != "tiny":
        cfg.n_layer, cfg.vocab_size = 1, 512
    sms = query()["sm_count"]
    if pos == 600:
        rt, _, nspan, _ = geometry.attn(M, pos, cfg.n_local_heads, cfg.n_head // cfg.n_local_heads, sms)
        assert (rt, nspan) == (1, 8)
    assert name == "tiny" or M < 64 or geometry.matrices(cfg, M, asym, sms)["qkv"][3] == 4
    eng = DecodeEngine(cfg, {k: v.cuda() for k, v in packing.synth_packed(cfg, 0, asym=asym).items()}, max_seq=pos + 512)
    eng.kc.normal_()
    eng.vc.normal_()
    toks = torch.randint(0, cfg.vocab_size, (M,), generator=torch.Generator().manual_seed(M), dtype=torch.int32).cuda()
    run = (lambda: eng.decode(17, 0).clone()) if M == 1 else (lambda: (eng.verify if M <= 64 else eng.prefill)(toks, pos)[0])
    ref = run()
    eng.check()
    for _ in range(8):
        eng.set_option(0, 0)
        run()
        assert eng.status()["code"] in (_lib.FB_OK, _lib.FB_ERR_TIMEOUT)
        eng.set_option(0, 4000000)
        again = run()
        eng.check()
        assert torch.equal(ref, again)
    eng.close()


def test_a_misaligned_feature_buffer_is_an_argument_error():
    """Features are stored 16 bytes at a time: a buffer that starts 2 bytes later is refused before any launch."""
    cfg = ModelArgs.from_name("tiny")
    eng = DecodeEngine(cfg, {k: v.cuda() for k, v in packing.synth_packed(cfg, 0).items()}, max_seq=32)
    tok, depth = (torch.arange(4, dtype=torch.int32, device="cuda") for _ in range(2))
    mask = torch.ones(4, 4, dtype=torch.uint8, device="cuda").tril()
    feat = torch.full((4 * cfg.dim + 8,), 7.0, dtype=torch.bfloat16, device="cuda")
    p = [ctypes.c_void_p(t.data_ptr()) for t in (tok, depth, mask)]
    for at in (2, 8):
        out = ctypes.c_void_p(feat.data_ptr() + at)
        assert eng.lib.fb_verify(eng._ctx, p[0], None, p[1], p[2], 4, 0, None, out, None) == _lib.FB_ERR_ARG
        assert eng.lib.fb_prefill(eng._ctx, p[0], 4, 0, None, out, None) == _lib.FB_ERR_ARG
    torch.cuda.synchronize()
    assert bool((feat == 7.0).all())
    eng.close()


def test_positions_near_the_end_of_the_integers_are_out_of_range():
    """pos + M past 2^31 - 1: refused like every position behind the cache, for trees, prompts and single steps."""
    cfg = ModelArgs.from_name("tiny")
    eng = DecodeEngine(cfg, {k: v.cuda() for k, v in packing.synth_packed(cfg, 0).items()}, max_seq=128)
    for pos in (2 ** 31 - 1, 2 ** 31 - 20, 128, -1):
        for call in (lambda: eng.verify(list(range(30)), pos), lambda: eng.prefill(list(range(30)), pos), lambda: eng.decode(3, pos)):
            with pytest.raises(_lib.FlintError) as ei:
                call()
            assert ei.value.code == _lib.FB_ERR_RANGE
    eng.close()


@pytest.mark.parametrize("M", [5, 40, 70])
def test_weight_scales_far_apart_take_the_long_dequantisation(M):
    """Scales of one row 2^12 apart (every third group of every second row shrunk): blocks that the one-fma form cannot hold exactly, next
    to blocks that it can, in the tree GEMM (5, 40 tokens) and the prompt GEMM (70)."""
    cfg = ModelArgs.from_name("tiny")
    P = packing.synth_packed(cfg, 0)
    for k in ("qkv_s", "o_s", "gu_s", "d_s"):
        P[k] = P[k].clone()
        P[k][..., ::2, ::3] *= 2.0 ** -12
    orc, eng = _pair(cfg, 128, 6, P)
    toks = torch.randint(0, cfg.vocab_size, (M,), generator=torch.Generator().manual_seed(M)).tolist()
    ref = np.concatenate([orc.verify(toks[i:i + 40], 6 + i)[0] for i in range(0, M, 40)])
    lg, _ = (eng.prefill if M > 64 else eng.verify)(toks, 6)
    eng.check()
    assert np.abs(lg.cpu().numpy() - ref).max() < _tol(ref)
    eng.close()


@pytest.mark.parametrize("M", [1, 65, 127, 128, 129, 1024, 1025])
def test_prompt_pass_tile_and_chunk_edges(M):
    """Prompt passes around the 128-token tile and around the 1024 rows of one pass, behind 3 cached rows: logits of the last
    rows and every cache row against the oracle, which takes the prompt in pieces of 64."""
    cfg = ModelArgs.from_name("tiny")
    cfg.n_layer = 2
    orc, eng = _pair(cfg, M + 8, 3)
    toks = torch.randint(0, cfg.vocab_size, (M,), generator=torch.Generator().manual_seed(M)).tolist()
    for i in range(0, M, 64):
        ref, _ = orc.verify(toks[i:i + 64], 3 + i)
    lg, _ = eng.prefill(toks, 3)
    eng.check()
    n = len(ref)
    assert np.abs(lg[M - n:].cpu().numpy() - ref).max() < _tol(ref)
    for dev, host in ((eng.kc, orc.kc), (eng.vc, orc.vc)):
        assert np.abs(_f32(dev[:, 3:3 + M]) - O.bf16_to_f32(host[:, 3:3 + M])).max() < 0.05
    eng.close()


def _prompt_against_oracle(cfg, M, asym=False):
    """Logits of all rows and every cache row of a prompt behind 3 cached rows; the oracle takes it in pieces of 64."""
    orc, eng = _pair(cfg, M + 8, 3, packing.synth_packed(cfg, 0, asym=asym))
    toks = torch.randint(0, cfg.vocab_size, (M,), generator=torch.Generator().manual_seed(M)).tolist()
    ref = np.concatenate([orc.verify(toks[i:i + 64], 3 + i)[0] for i in range(0, M, 64)])
    lg, _ = eng.prefill(toks, 3)
    eng.check()
    assert np.abs(lg.cpu().numpy() - ref).max() < _tol(ref)
    for dev, host in ((eng.kc, orc.kc), (eng.vc, orc.vc)):
        assert np.abs(_f32(dev[:, 3:3 + M]) - O.bf16_to_f32(host[:, 3:3 + M])).max() < 0.05
    eng.close()


@pytest.mark.parametrize("asym", [False, True])
@pytest.mark.parametrize("M,splits", [(65, (4, 4, 4)), (128, (4, 4, 4)), (129, (2, 4, 4)), (300, (2, 2, 2))])
def test_prompt_tiles_with_split_k(M, splits, asym):
    """Short prompts on a shape with few row blocks (24 / 16 / 16 of QKV, O, down; 4 of the LM head): one, two and three token tiles run as clusters
    of four and of two, one of them with tokens in only part of its ranks."""
    cfg = ModelArgs.from_name("llama-1b-class")
    cfg.n_layer, cfg.vocab_size = 1, 512
    g = geometry.matrices(cfg, M, asym, query()["sm_count"])
    assert tuple(g[n][3] for n in ("qkv", "o", "d")) == splits and g["lm"][3] == 4 and g["o"][2] == -(-M // 128)
    _prompt_against_oracle(cfg, M, asym)


@pytest.mark.parametrize("asym", [False, True])
def test_prompt_tiles_with_split_k_of_gate_and_up(asym):
    """A model whose 32 gate/up row blocks are few enough for a prompt's SwiGLU to run over a cluster. No built-in shape is one: this runs on a library
    built with FLINT_B200_EXTRA_SHAPES="2048,2048,2048,64,4"."""
    cfg = ModelArgs(block_size=256, vocab_size=512, n_layer=1, n_head=32, n_local_heads=8, dim=2048, intermediate_size=2048)
    try:
        DecodeEngine(cfg, {k: v.cuda() for k, v in packing.synth_packed(cfg, 0, asym=asym).items()}, max_seq=8).close()
    except _lib.FlintError as e:
        assert e.code == _lib.FB_ERR_SHAPE
        pytest.skip("library built without the shape 2048,2048,2048,64,4")
    for M, splits in ((65, 4), (81, 4), (128, 4), (129, 2)):
        assert geometry.matrices(cfg, M, asym, query()["sm_count"])["gu"][2:] == (-(-M // 128), splits)
        _prompt_against_oracle(cfg, M, asym)


@pytest.mark.parametrize("name,vocab,M,wide", [
    ("llama-1b-class", 512, 161, "gu"), ("llama-1b-class", 512, 192, "gu"), ("llama-1b-class", 512, 257, "gu"), ("llama-1b-class", 512, 384, "gu"),
    ("llama-1b-class", 512, 513, "gu"), ("llama-1b-class", 512, 900, "qkv gu"), ("llama-1b-class", 20000, 161, "gu lm"),
    ("llama-1b-class", 20000, 700, "gu lm"), ("granite-3b-class", 10000, 900, "o gu d lm"), ("granite-3b-class", 512, 1000, "o d"),
    ("llama-8b-class", 512, 520, "qkv o gu d")])
def test_prompt_tiles_of_192_tokens(name, vocab, M, wide):
    """Prompts some of whose matrices take fewer rounds as 192-token tiles, every epilogue among them: a tile not quite and just full, the first
    tokens of a second and a third tile, tiles cut evenly into halves of 96 and less; the LM head with a last row block that is not full."""
    cfg = ModelArgs.from_name(name)
    cfg.n_layer, cfg.vocab_size = 1, vocab
    g = geometry.matrices(cfg, M, sms=query()["sm_count"])
    assert [n for n in g if g[n][0] == 192] == wide.split()
    _prompt_against_oracle(cfg, M)


@pytest.mark.parametrize("pos,Ms", [(127, (4,)), (128, (14,)), (129, (26,)), (1000, (4, 14, 26, 61)), (3001, (4, 26))])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_verify_attention_over_spans_of_every_geometry(name, pos, Ms):
    """Trees behind cached prefixes for every head geometry, 40 / 8 heads (whose row tiles cut a token's heads) and heads of 128 among them: one, two
    and four row tiles a CTA, clusters of two to eight, the first stages requested ahead of the wait and, at 3001, more than those; a random
    ancestor mask."""
    cfg = ModelArgs.from_name(name)
    cfg.n_layer, cfg.vocab_size = 1, 512
    if pos == 1000:
        r = cfg.n_head // cfg.n_local_heads
        geo = [geometry.attn(M, pos, cfg.n_local_heads, r, query()["sm_count"]) for M in Ms]
        assert [(g[0], g[2]) for g in geo] == ([(1, 8), (1, 4), (2, 4), (4, 4)] if r == 4 else [(1, 4), (2, 4), (4, 4), (4, 2)])
    orc, eng = _pair(cfg, pos + 64, pos)
    for M in Ms:
        g = torch.Generator().manual_seed(M)
        toks = torch.randint(0, cfg.vocab_size, (M,), generator=g).tolist()
        parent = [-1] + [int(torch.randint(0, i, (1,), generator=g)) for i in range(1, M)]
        mask = tree_mask(parent)
        depth = mask.sum(1).astype(np.int32) - 1
        ref, _ = orc.verify(toks, pos, depth, mask)
        lg, _ = eng.verify(toks, pos, torch.from_numpy(depth), torch.from_numpy(mask))
        eng.check()
        assert np.abs(lg.cpu().numpy() - ref).max() < _tol(ref)
        assert np.abs(_f32(eng.kc[:, pos:pos + M]) - O.bf16_to_f32(orc.kc[:, pos:pos + M])).max() < 0.05
    eng.close()


@pytest.mark.parametrize("vocab", [1, 31, 4096, 8200, 32768, 49160, 128256, 300001])
def test_token_choice_over_every_split_of_a_row(vocab):
    """Rows on one, two, four and eight CTAs, slices that fit the registers and slices that do not, ragged ends: the arg-max
    (first index on a tie at the two ends of the row), draws confined to the top-k entries, and the k = 1 draw."""
    cfg = ModelArgs.from_name("tiny")
    eng = DecodeEngine(cfg, {k: v.cuda() for k, v in packing.synth_packed(cfg, 0).items()}, max_seq=8)
    lg = torch.randn(3, vocab, generator=torch.Generator().manual_seed(vocab)).cuda()
    lg[1, 0] = lg[1, vocab - 1] = 9.0
    lg[2, vocab - 1] = 11.0
    assert eng.sample(lg, 0.0).tolist() == [int(lg[0].argmax()), 0, vocab - 1]
    assert eng.sample(lg[2], 0.8, 1, seed=5).tolist() == [vocab - 1]
    for k in (2, 50):
        n = 256
        out = torch.empty(n, dtype=torch.int32, device="cuda")
        _lib.check(eng.lib.fb_sample(ctypes.c_void_p(lg.data_ptr()), vocab, n, 0, 1.0, k, 3, 0, ctypes.c_void_p(out.data_ptr()), None), "fb_sample")
        p = sample_probs(lg[0].cpu().numpy(), 1.0, k)
        assert np.all(p[out.cpu().numpy()] > 0)
        if vocab > 50:
            assert len(set(out.tolist())) > 1
    eng.close()


def _sample(eng, lg, vocab, rows, top_k, counter):
    out = torch.full((rows,), -1, dtype=torch.int32, device="cuda")
    _lib.check(eng.lib.fb_sample(ctypes.c_void_p(lg.data_ptr()), vocab, rows, 0, 1.0, top_k, 3, counter, ctypes.c_void_p(out.data_ptr()), None),
               "fb_sample")
    return out


@pytest.mark.parametrize("vocab,top_k", [(300, 0), (300, 7), (8200, 0)])
def test_token_choice_of_more_rows_than_a_grid_has_in_y(vocab, top_k):
    """70 000 draws from one vector (stride 0) in one call. Row r draws from stream (seed, counter + r): every row equals a
    short call that starts at its counter, below, across and above row 65 535."""
    cfg = ModelArgs.from_name("tiny")
    eng = DecodeEngine(cfg, {k: v.cuda() for k, v in packing.synth_packed(cfg, 0).items()}, max_seq=8)
    lg = torch.randn(vocab, generator=torch.Generator().manual_seed(vocab)).cuda()
    out = _sample(eng, lg, vocab, 70000, top_k, 11)
    for r0 in (0, 65520, 69970):
        assert torch.equal(out[r0:r0 + 30], _sample(eng, lg, vocab, 30, top_k, 11 + r0))
    eng.close()


@pytest.mark.parametrize("vocab", [8200, 16390, 49160, 300001])
@pytest.mark.parametrize("temperature,top_k", [(1.0, 0), (0.7, 5), (1.5, 400)])
def test_sampled_frequencies_of_rows_on_several_ctas(vocab, temperature, top_k):
    """20 000 draws from one row that 2, 4 or 8 CTAs share, with a run of equal values at the top-k threshold that crosses a slice boundary:
    nothing outside the support, every frequency within 5 sigma (a threshold that keeps too few entries loses whole tokens)."""
    cfg = ModelArgs.from_name("tiny")
    eng = DecodeEngine(cfg, {k: v.cuda() for k, v in packing.synth_packed(cfg, 0).items()}, max_seq=8)
    lg = torch.randn(vocab, generator=torch.Generator().manual_seed(vocab + top_k)) * 2.0
    if top_k:
        kth = torch.topk(lg, top_k).values[-1]
        lg[vocab // 2 - 3:vocab // 2 + 3] = kth
    n = 20000
    lg = lg.cuda()
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    _lib.check(eng.lib.fb_sample(ctypes.c_void_p(lg.data_ptr()), vocab, n, 0, temperature, top_k, 123, 0, ctypes.c_void_p(out.data_ptr()), None),
               "fb_sample")
    counts = np.bincount(out.cpu().numpy(), minlength=vocab).astype(np.float64)
    p = sample_probs(lg.cpu().numpy(), temperature, top_k)
    assert counts.size == vocab and counts[p == 0].sum() == 0
    sigma = np.sqrt(n * p * (1 - p)) + 1.0
    assert np.all(np.abs(counts - n * p) < 5 * sigma), float(np.max(np.abs(counts - n * p) / sigma))
    eng.close()


@pytest.mark.parametrize("top_b", [1, 3, 16])
@pytest.mark.parametrize("vocab", [1000, 8200, 16390, 49160, 140000])
def test_token_head_order_over_every_split_of_a_row(vocab, top_b):
    """The B best tokens of rows on 1, 2, 4 and 8 CTAs, slices in registers and slices read again (140 000). One-hot feature rows make
    the logits exactly 8 x one column of the embedding table, so the order (value descending, first index on ties) is known: a row of normal
    values, whose bf16 ties are many; one whose winners all lie in one slice; one whose winners are ties on both sides of every slice
    boundary; a constant row."""
    dim = 64
    m = seeded_draft(dim, 1, 64, seed=1, rope_base=10000.0)
    g = torch.Generator().manual_seed(vocab)
    embed = torch.randn(vocab, dim, generator=g).bfloat16()
    ctas = 1
    while ctas < 8 and vocab >= 8192 * ctas:
        ctas *= 2
    per = -(-vocab // ctas)
    embed[:, 1].clamp_(max=2.0)
    embed[per * (ctas - 1):per * (ctas - 1) + 20, 1] = torch.arange(20).bfloat16() / 4 + 4
    for c in range(1, ctas):
        embed[c * per - 2:c * per + 2, 2] = 6.0
    embed[:, 3] = 1.0
    m.bind_target(embed.cuda(), torch.ones(dim, dtype=torch.bfloat16, device="cuda"))
    m.setup_cache(8)
    rows = torch.zeros(4, dim, dtype=torch.bfloat16, device="cuda")
    rows[torch.arange(4), torch.arange(4)] = 8.0              # mean square 1: the norm leaves 8
    toks, scores = m.head(rows, top_b=top_b, want_scores=True)
    for r in range(4):
        v = 8.0 * embed[:, r].float().numpy()
        order = np.lexsort((np.arange(vocab), -v))[:top_b]
        assert toks[r].tolist() == order.tolist() and scores[r].tolist() == v[order].tolist()


@pytest.mark.parametrize("T", [1, 7, 8, 9, 16, 17, 33])
def test_draft_row_tile_edges(T):
    """The draft head's linears take 8 rows per MMA tile: below, at and above one, two and four tiles."""
    dim, nh, nkv, inter, vocab = 256, 8, 2, 512, 1000
    m = seeded_draft(dim, nh, inter, seed=5, rope_base=10000.0, n_kv=nkv, fuse=2)
    g = torch.Generator().manual_seed(T)
    embed = (torch.randn(vocab, dim, generator=g) * 0.5).bfloat16().cuda()
    nf = (torch.rand(dim, generator=g) + 0.5).bfloat16().cuda()
    m.bind_target(embed, nf, logits_scaling=4.0)
    m.setup_cache(48)
    orc = DraftOracle({k: _f32(v) for k, v in m._w.items()}, nh, 10000.0, max_roll=48, n_kv=nkv)
    feat = torch.randn(T, 2 * dim, generator=g).bfloat16().cuda()
    toks = torch.randint(-1, vocab, (T,), generator=g).to(torch.int32)
    pos = torch.arange(T, dtype=torch.int32)
    out = m(feat, None, pos.cuda(), input_pos=pos.cuda(), tokens=toks.cuda())
    emb = np.stack([_f32(embed[t]) if t >= 0 else np.zeros(dim, np.float32) for t in toks.tolist()])
    ref = orc.forward(_f32(feat), emb, pos.numpy(), slots=np.arange(T))
    assert np.abs(_f32(out) - ref).max() <= 2e-2 * np.abs(ref).max()         # as in the rollout test: bf16 between the layers
    t_dev, s_dev = m.head(out[:16], top_b=3, want_scores=True)          # at most 16 rows a call
    lg = orc.head_logits(_f32(out[:16]), _f32(nf), _f32(embed), 4.0)              # the head alone: same input rows on both sides
    top = -np.sort(-lg, axis=1)[:, :3]
    assert np.abs(s_dev.cpu().numpy() - top).max() <= 2.0 ** -6 * np.abs(lg).max()      # bf16 logits: 2^-9, a near-tie may swap ranks
    assert np.all(np.take_along_axis(lg, t_dev.cpu().numpy().astype(np.int64), 1) >= top[:, 2:] - 2.0 ** -6 * np.abs(lg).max())


@pytest.mark.parametrize("T", [1, 8, 16, 33])
@pytest.mark.parametrize("dim,inter", [(256, 1024), (256, 1544), (256, 2048), (1024, 1032), (1536, 1032)])
def test_draft_linears_with_split_k(T, dim, inter):
    """Linears whose K goes over a cluster. 256 wide: the merge (K = 1024) over two CTAs, the down projection over two or three, one of them with a K that
    is no multiple of a chunk. 1024 and 1536 wide: q, k and v in one grid, the SwiGLU pair, O and the last linear too, over two and three CTAs."""
    nh, nkv, vocab, sms = dim // 128 * 4, dim // 128, 1000, query()["sm_count"]
    kv = nkv * (dim // nh)
    for n in {min(T, 32), T - 32 if T > 32 else T}:
        ks = [geometry.draft(rows, k, n, pair, sms) for rows, k, pair in (((dim,), 4 * dim, False), ((dim, kv, kv), dim, False), ((inter,), dim, True))]
        assert ks == ([2, 1, 1] if dim == 256 else [3, 2, 2] if dim == 1024 else [3, 3, 3])
    m = seeded_draft(dim, nh, inter, seed=5, rope_base=10000.0, n_kv=nkv, fuse=3)
    g = torch.Generator().manual_seed(T)
    m.bind_target((torch.randn(vocab, dim, generator=g) * 0.5).bfloat16().cuda(), torch.ones(dim, dtype=torch.bfloat16).cuda(), 1.0)
    m.setup_cache(48)
    orc = DraftOracle({k: _f32(v) for k, v in m._w.items()}, nh, 10000.0, max_roll=48, n_kv=nkv)
    feat, emb = (torch.randn(T, n * dim, generator=g).bfloat16().cuda() for n in (3, 1))
    pos = torch.arange(T, dtype=torch.int32)
    out = m(feat, emb, pos.cuda(), input_pos=pos.cuda())
    ref = orc.forward(_f32(feat), _f32(emb), pos.numpy(), slots=np.arange(T))
    assert np.abs(_f32(out) - ref).max() <= 2e-2 * np.abs(ref).max()         # as above


@pytest.mark.parametrize("T", [1, 12, 40])
def test_draft_token_ids_outside_the_table_are_zero_rows(T):
    """Ids at and past the vocabulary, like negative ones, read no table row: the bits of a call whose embeddings are zeros there."""
    dim, vocab = 256, 1000
    m = seeded_draft(dim, 4, 512, seed=5, rope_base=10000.0)
    g = torch.Generator().manual_seed(T)
    embed = torch.randn(vocab, dim, generator=g).bfloat16().cuda()
    m.bind_target(embed, torch.ones(dim, dtype=torch.bfloat16, device="cuda"))
    m.setup_cache(48)
    feat = torch.randn(T, dim, generator=g).bfloat16().cuda()
    toks = torch.randint(0, vocab, (T,), generator=g, dtype=torch.int32)
    bad = torch.arange(T) % 3 == 0
    toks[bad] = torch.tensor([vocab, -1, 2 ** 31 - 1, vocab + 7, -2 ** 31], dtype=torch.int32).repeat(T)[:int(bad.sum())]
    emb = embed[toks.clamp(0, vocab - 1).long().cuda()]
    emb[bad.cuda()] = 0
    pos = torch.arange(T, dtype=torch.int32, device="cuda")
    assert torch.equal(m(feat, None, pos, input_pos=pos, tokens=toks.cuda()), m(feat, emb, pos, input_pos=pos))


@pytest.mark.parametrize("slots", [12284, 20000])
def test_draft_attention_over_a_large_cache(slots):
    """A draft head whose score vector alone fills (12 284 slots), or exceeds, the 48 KB of shared memory that a kernel has without asking:
    the same bits as with a small cache."""
    dim, outs = 128, []
    g = torch.Generator().manual_seed(4)
    feat, emb = (torch.randn(5, dim, generator=g).bfloat16().cuda() for _ in range(2))
    pos = torch.arange(5, dtype=torch.int32, device="cuda")
    for n in (8, slots):
        m = seeded_draft(dim, 2, 256, seed=5, rope_base=10000.0)
        m.bind_target(torch.zeros(16, dim, dtype=torch.bfloat16, device="cuda"), torch.ones(dim, dtype=torch.bfloat16, device="cuda"))
        m.setup_cache(n)
        outs.append(m(feat, emb, pos, input_pos=pos))
    assert torch.equal(outs[0], outs[1])


def test_weights_written_just_before_a_call_are_the_ones_it_uses():
    """The caller's weights are bound by pointer. A matrix product that writes the draft's merge matrix or its embedding table, and an
    elementwise kernel that writes the target's norms, directly before a call on the same stream: the call gives what a call
    long after them gives, bit for bit."""
    dim = 512
    m = seeded_draft(dim, 8, 1024, seed=5, rope_base=10000.0)
    g = torch.Generator().manual_seed(2)
    embed = torch.randn(4096, dim, generator=g).bfloat16().cuda()
    m.bind_target(embed, torch.ones(dim, dtype=torch.bfloat16, device="cuda"))
    m.setup_cache(48)
    feat = torch.randn(40, dim, generator=g).bfloat16().cuda()
    emb, pos = torch.randn(40, dim, generator=g).bfloat16().cuda(), torch.arange(40, dtype=torch.int32, device="cuda")
    cfg = ModelArgs.from_name("tiny")
    eng = DecodeEngine(cfg, {k: v.cuda() for k, v in packing.synth_packed(cfg, 0).items()}, max_seq=128)
    a = [torch.randn(n, 2048, generator=g).bfloat16().cuda() * 0.02 for n in (dim, 4096)]
    b = [torch.randn(2048, n, generator=g).bfloat16().cuda() for n in (2 * dim, dim)]
    for i in range(20):
        torch.mm(a[0], b[0] * (1 + i), out=m._w["merge.weight"])
        out = m(feat, emb, pos, input_pos=pos)
        torch.mm(a[1], b[1] * (1 + i), out=embed)
        toks, scores = m.head(feat[:3], top_b=4, want_scores=True)
        for k in ("n1", "n2", "nf"):
            eng._keep[k].fill_(1.0 + 0.25 * i)
        lg, ft = eng.verify(list(range(i, i + 20)), 0)
        torch.cuda.synchronize()
        assert torch.equal(out, m(feat, emb, pos, input_pos=pos))
        toks2, scores2 = m.head(feat[:3], top_b=4, want_scores=True)
        assert torch.equal(toks, toks2) and torch.equal(scores, scores2)
        lg2, ft2 = eng.verify(list(range(i, i + 20)), 0)
        assert torch.equal(lg, lg2) and torch.equal(ft, ft2)
        assert i == 0 or not (torch.equal(out, last[0]) or torch.equal(scores, last[1]) or torch.equal(lg, last[2]))
        last = (out, scores, lg)
    eng.check()
    eng.close()
