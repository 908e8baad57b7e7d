"""GPU: the SwiGLU output of the M-token passes, bit by bit.

One layer whose matrices make every intermediate exact, whatever the order of a sum: attention off (scales of zero), one nonzero weight
in every gate, up and down row, embedding rows that are permutations of one multiset of 7-bit values with mean square 2^20 (their norm is a
division by 2^10), and two rows of the down matrix so large that the final norm is a division by 2^50. The feature row then holds the SwiGLU
outputs themselves, which have to be bf16((g / (1 + e^-g)) * u) with the division that `/` means, for trees and prompts as in the decode kernel."""
import numpy as np
import pytest
import torch

from flint_b200 import packing
from flint_b200.config import ModelArgs
from flint_b200.engine import DecodeEngine

pytestmark = pytest.mark.gpu

_SILU = """
extern "C" __global__ void silu(const float* g, float* exact, float* approx, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float d = 1.0f + __expf(-g[i]);
  exact[i] = __fdiv_rn(g[i], d);
  approx[i] = __fdividef(g[i], d);
}
"""


def _rows(D, n, rng):
    """n permutations (component 0 fixed, random signs) of D integers in 16..127 whose squares sum to D * 64^2; component 0 is 64."""
    k = np.concatenate([[64], rng.integers(20, 101, D - 1)]).astype(np.int64)
    while (off := int((k * k).sum()) - D * 4096) != 0:
        i, step = int(rng.integers(1, D)), -1 if off > 0 else 1
        new = k[i] + step
        if 16 <= new <= 127 and (abs(off + new * new - k[i] * k[i]) < abs(off) or rng.random() < 0.1):
            k[i] = new
    out = np.empty((n, D), np.int64)
    for r in range(n):
        out[r, 0] = 64
        out[r, 1:] = rng.permutation(k[1:]) * rng.choice((-1, 1), D - 1)
    return out


def _one_hot(rows, cols, at, sign):
    """int32 words of a matrix whose row r is sign[r] at column at[r] and zero (nibble 8) elsewhere."""
    nib = np.full((rows, cols), 8, np.uint32)
    nib[np.arange(rows), at] = 8 + sign
    w = (nib.reshape(rows, cols // 8, 8) << (4 * np.arange(8, dtype=np.uint32))).sum(-1, dtype=np.uint32)
    return torch.from_numpy(w.view(np.int32))


def build(cfg, rng, tail):
    """(packed, embedding rows / 1024, column and sign and scale of every gate and up row, down's columns, power of two of the feature).
    Gates and ups of +-1/8 .. +-4; `tail`: gates of -15 .. -6, the pair (-15, 1.3671875) among them, whose result an approximate division
    rounds the other way. Rows 0 and 1: silu(64) * 1 = 64, or silu(16) * 1 = 16. All |act| stay exact in fp16 under the token's bound."""
    D, F = cfg.dim, cfg.ffn_padded
    P = packing.synth_packed(cfg, 0)
    for k in ("qkv_s", "o_s"):
        P[k].zero_()
    col, sign = rng.integers(1, D, (2, F)), rng.choice((-1, 1), (2, F))
    scale = rng.uniform(0.5, 2.0, (2, F))
    if tail:
        col[:], sign[0], sign[1] = 0, -1, 1
        scale = np.stack([rng.uniform(6.0, 15.0, F), rng.uniform(1.0, 1.98, F)])
        scale[0, 2:66], scale[1, 2:66] = 15.0, 1.3671875
    col[:, :2], sign[:, :2] = 0, 1
    scale[0, :2], scale[1, :2] = 16.0 if tail else 64.0, 1.0
    scale = torch.from_numpy(scale).bfloat16()
    P["gu_q"][0] = _one_hot(2 * F, D, col.reshape(-1), sign.reshape(-1))
    P["gu_s"][0] = scale.reshape(-1, 1).expand(-1, D // 128)
    pick = np.concatenate([np.arange(66), 66 + rng.permutation(F - 66)[:D - 66]])
    down = 44 if tail else 30
    P["d_q"][0] = _one_hot(D, F, pick, np.ones(D, np.int64))
    P["d_s"][0] = 2.0 ** down
    P["d_s"][0, :2] = 2.0 ** (50 if tail else 48)
    x = torch.from_numpy(_rows(D, cfg.vocab_size, rng)).float() / 64
    P["embed"].copy_(x * 1024)
    return P, x, torch.from_numpy(col), torch.from_numpy(sign), scale.float(), torch.from_numpy(pick), 2.0 ** (50 - down)


def gates_and_ups(x, col, sign, scale):
    return [(x[:, col[i]] * (sign[i] * scale[i])).bfloat16().float().contiguous() for i in range(2)]


@pytest.mark.parametrize("tail", [False, True])
@pytest.mark.parametrize("M", [16, 32, 64, 100, 700, 1024])
def test_swiglu_of_the_token_passes_is_the_exact_expression(M, tail):
    cfg = ModelArgs.from_name("tiny")
    cfg.n_layer, cfg.vocab_size = 1, 2048
    P, x, col, sign, scale, pick, back = build(cfg, np.random.default_rng(M), tail)
    eng = DecodeEngine(cfg, {k: v.cuda() for k, v in P.items()}, max_seq=1024)
    g, u = gates_and_ups(x.cuda(), col.cuda(), sign.cuda(), scale.cuda())
    exact, approx = torch.empty_like(g), torch.empty_like(g)
    torch.cuda._compile_kernel(_SILU, "silu")(grid=(-(-g.numel() // 256), 1, 1), block=(256, 1, 1), args=(g, exact, approx, g.numel()))
    want, other = ((s * u).bfloat16()[:, pick.cuda()] for s in (exact, approx))
    assert not tail or bool((want[:, 2:66] != other[:, 2:66]).all())       # the inputs tell the two divisions apart
    for t0 in range(0, cfg.vocab_size, M):
        tok = torch.arange(t0, min(cfg.vocab_size, t0 + M), dtype=torch.int32, device="cuda")
        got = (eng.verify if M <= 64 else eng.prefill)(tok, 0, want_logits=False)[1]
        assert torch.equal(got[:, 2:].float() * back, want[t0:t0 + M, 2:].float())
    eng.check()
    eng.close()
