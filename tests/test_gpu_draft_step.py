"""GPU: a single draft row (norms inside the linears, rotation inside the attention) gives what the same row gives as one of two rows."""
import pytest
import torch

from flint_b200.draft import seeded_draft

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,nh,nkv", [(512, 8, 2), (640, 8, 8), (4096, 32, 8), (4104, 9, 3)])
@pytest.mark.parametrize("slot", [0, 1, 15, 16])
def test_one_row_like_a_row_of_two(dim, nh, nkv, slot):
    """Same operations in the same order: equal bits, in the output and in the cache that the next row reads. 4104: a row that does not fit the registers. Slot
    16 of 16: outside the cache, no write and no rotation."""
    g = torch.Generator(device="cuda").manual_seed(dim + slot)
    feat = torch.randn(18, dim, generator=g, device="cuda").bfloat16()
    emb = torch.randn(18, dim, generator=g, device="cuda").bfloat16()
    outs = []
    for pair in (False, True):
        m = seeded_draft(dim, nh, 256, seed=1, n_kv=nkv)
        m.bind_target(torch.zeros(64, dim, device="cuda", dtype=torch.bfloat16), torch.ones(dim, device="cuda", dtype=torch.bfloat16), 1.0)
        m.setup_cache(16)
        s = torch.arange(16, dtype=torch.int32, device="cuda")
        m(feat[:16], emb[:16], s, input_pos=s)
        at = torch.tensor([slot], dtype=torch.int32, device="cuda")
        last = torch.tensor([15], dtype=torch.int32, device="cuda")
        if pair:                                  # the second row lies in a slot that the first does not see
            other = torch.tensor([slot, -1], dtype=torch.int32, device="cuda")
            a = m(feat[16:], emb[16:], other.clamp_min(0), input_pos=other)[:1]
        else:
            a = m(feat[16:17], emb[16:17], at, input_pos=at)
        b = m(feat[17:18], emb[17:18], last, input_pos=last)
        outs.append((a.clone(), b.clone()))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
