"""CPU: the launch geometry of the M-token passes and of the draft linears over the whole range of sizes: every token has a tile and no tile is empty,
clusters are of sizes that the kernels handle and are resident at once, and each CTA of a split has work."""
import geometry as G
import pytest

from flint_b200.config import ModelArgs

MODELS = ("tiny", "llama-1b-class", "granite-3b-class", "granite-4.1-3b", "llama-8b-class")


@pytest.mark.parametrize("asym", [False, True])
@pytest.mark.parametrize("sms", [132, 148, 160])
@pytest.mark.parametrize("name", MODELS)
def test_gemm_tiles_cover_the_tokens_and_splits_have_work(name, sms, asym):
    cfg = ModelArgs.from_name(name)
    ks = dict(qkv=cfg.dim, o=cfg.n_head * cfg.head_dim, gu=cfg.dim, d=cfg.ffn_padded, lm=cfg.dim)
    rows = dict(qkv=cfg.qkv_rows, o=cfg.dim, gu=2 * cfg.ffn_padded, d=cfg.dim, lm=cfg.vocab_size)
    for M in range(1, 1025):
        for n, (nt, ntok, ntile, ns) in G.matrices(cfg, M, asym, sms).items():
            assert nt in ((16, 32, 64) if M <= 64 else ((128,) if asym else (128, 192)))
            assert ntok % 16 == 0 and ntok <= nt and (ntile - 1) * ntok < M <= ntile * ntok
            assert ntile == 1 or nt >= 128
            ctas, per_sm = -(-rows[n] // 128) * ntile * ns, 2 if nt <= 64 else 1
            assert ns in ((1, 2, 4, 8) if nt <= 64 else (1, 2, 4) if nt == 128 else (1,))
            if ns > 1:
                assert ctas <= per_sm * sms and ks[n] // 128 // ns >= (2 if nt <= 64 else 4) and nt // ns >= 2


@pytest.mark.parametrize("n_kv,r", [(2, 4), (8, 4), (8, 5)])
def test_attention_spans_cover_the_positions(n_kv, r):
    for M in (*range(1, 65), 65, 100, 128, 300, 725, 1024):
        for pos in (0, 1, 63, 64, 127, 128, 129, 500, 1000, 3001, 32768):
            rt, groups, nspan, span = G.attn(M, pos, n_kv, r)
            tiles = -(-M * r // 16)
            assert rt in (1, 2, 4) and (groups - 1) * rt < tiles <= groups * rt
            assert nspan in (1, 2, 4, 8) and span % 64 == 0 and nspan * span >= pos + M
            assert nspan == 1 or groups * n_kv * nspan <= (98 if nspan == 8 else 148)


def test_draft_splits_are_resident_and_leave_every_warp_two_chunks():
    for rows in (16, 256, 1024, 1032, 2560, 8192, 49160):
        for k in (64, 256, 1024, 1536, 1544, 2560, 5120, 8192):
            for T in (1, 8, 9, 16, 17, 32):
                for pair in (False, True):
                    ks = G.draft((rows,), k, T, pair)
                    blocks = -(-rows // (16 if T <= 8 or pair else 32))
                    assert 1 <= ks <= 3
                    assert ks == 1 or (blocks * ks <= 148 * (3 if T <= 8 else 2) and -(-k // 32) >= 16 * ks)
