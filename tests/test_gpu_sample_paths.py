"""GPU: the two selections of the token choice (the list of the few values above the k-th largest warp maximum; the radix select) draw the same tokens."""
import pytest
import torch

from flint_b200 import packing
from flint_b200.config import ModelArgs
from flint_b200.engine import DecodeEngine

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    cfg = ModelArgs.from_name("tiny")
    return DecodeEngine(cfg, packing.synth_packed(cfg, 0, device="cuda"), max_seq=32)


def _rows(kind, rows, vocab):
    g = torch.Generator(device="cuda").manual_seed(vocab + rows)
    lg = torch.randn(rows, vocab, generator=g, device="cuda") * 2.5
    if kind == "ties":
        lg = (lg * 2).round() / 2
    elif kind == "flat":
        lg.fill_(1.5)
    elif kind == "one":                       # a single finite value
        lg.fill_(float("-inf"))
        lg[:, vocab // 3] = 1.0
    elif kind == "mixed":                     # +-0, infinities and the lowest value among the rest
        lg[:, ::7] = float("-inf")
        lg[:, 3::11] = -0.0
        lg[:, 5::13] = 0.0
        lg[:, 6::17] = torch.finfo(torch.float32).min
    elif kind == "sorted":                    # all large values in one CTA, one warp
        lg = lg.sort(dim=1, descending=True).values.contiguous()
    return lg


@pytest.mark.parametrize("kind", ["normal", "ties", "flat", "one", "mixed", "sorted"])
@pytest.mark.parametrize("vocab", [700, 4097, 8192, 49160, 128256, 131073, 200000])
def test_top_k_of_list_and_radix_select(eng, vocab, kind):
    """k up to 4/5 of the row's warps takes the list, more the radix select. A row whose entries below the k-th largest value are minus infinity is, for the
    radix select, the same distribution with the same noise: both calls have to return the same tokens. One CTA (32 warps) to eight, rows read
    once and several times, ties that overflow the list."""
    ctas = 1
    while ctas < 8 and vocab >= 8192 * ctas:
        ctas *= 2
    most = ctas * 32 * 4 // 5
    lg = _rows(kind, 3, vocab)
    for k in (1, 2, most // 2, most, most + 1):
        kept = lg.clone()
        kept[kept < kept.topk(k, dim=1).values[:, -1:]] = float("-inf")
        got = eng.sample(lg, 0.8, k, seed=9, counter=2)
        want = eng.sample(kept, 0.8, None, seed=9, counter=2)
        assert got.tolist() == want.tolist()
