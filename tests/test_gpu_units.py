"""GPU: how the tile product cuts a CTA's rows into units (whole tiles, chunks of long rows, slices by rounds) and how it represents activations."""
import ctypes

import numpy as np
import pytest
import torch

from flint_b200 import _lib, packing
from flint_b200.engine import query
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _gemv(q, s, z, x):
    lib, rows, k = _lib.load(), q.shape[0], q.shape[1] * 8
    dq, ds, dz, dx = q.cuda(), s.cuda(), None if z is None else z.cuda(), x.cuda()
    st = torch.empty(lib.fb_stream_bytes(rows, k, int(z is not None)) + 16, dtype=torch.uint8, device="cuda")
    _lib.check(lib.fb_repack(_p(dq), _p(ds), None if z is None else _p(dz), rows, k, 0, 0, 0, _p(st), None), "fb_repack")
    y = torch.full((rows,), 7.0, device="cuda")
    status = torch.zeros(8, dtype=torch.int32, device="cuda")
    _lib.check(lib.fb_gemv(_p(st), rows, k, int(z is not None), 0, 0, 0, _p(dx), _p(y), _p(status), None), "fb_gemv")
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    return y.cpu().numpy()


def _matrix(rows, k, asym, seed):
    g = torch.Generator().manual_seed(seed)
    q = torch.randint(-2 ** 31, 2 ** 31 - 1, (rows, k // 8), generator=g, dtype=torch.int64).to(torch.int32)
    s = (torch.rand(rows, k // 128, generator=g) * 0.01 + 1e-4).bfloat16()
    return q, s, (torch.randn(rows, k // 128, generator=g) * 0.01).bfloat16() if asym else None


@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 7, 8, 15])
@pytest.mark.parametrize("k,asym", [(2048, False), (2560, True), (8192, False), (14336, True), (1408, False)])
def test_every_number_of_tiles_a_cta(k, asym, tiles):
    """1 .. 15 tiles of a CTA (8 rows; 16 where k has an odd number of groups): tiles in 14, 7, 4, 3, 2 and no slices, tiles of 2 and 7 chunks, more chunks
    than warps. The rows behind the last whole tile are plain ones here (tiles with padding: the vocabulary test of the decode step). fp32 sums of k
    exact products in any order differ from the oracle's by less than 2e-5 of the largest result (64 roundings of 2^-24 each and the oracle's own)."""
    rt = 8 if (k // 128) % 2 == 0 else 16
    rows = query(torch.cuda.current_device())["sm_count"] * rt * tiles - 3
    q, s, z = _matrix(rows, k, asym, k + tiles)
    x = torch.randn(k, generator=torch.Generator().manual_seed(1)).bfloat16()
    got, ref = _gemv(q, s, z, x), O.c_gemv(q, s, z, x)[0]
    assert np.abs(got - ref).max() < 2e-5 * np.abs(ref).max()


@pytest.mark.parametrize("k", [512, 640])
def test_activations_far_apart_in_a_group(k):
    """One element of a group 2^21 above the rest: every bf16 element is still exact in the integers that are multiplied, so rows whose weight of the
    large element is zero (nibble 8) have exactly the small elements' sum. (q, s): small integers, so fp32 holds every sum."""
    rows = 64
    q, _, _ = _matrix(rows, k, False, 3)
    q[:, 0] = (q[:, 0] & ~0xF) | 8
    s = torch.ones(rows, k // 128).bfloat16()
    x = torch.randint(1, 8, (k,), generator=torch.Generator().manual_seed(2)).float()
    x[0] = 2.0 ** 22
    got = _gemv(q, s, None, x.bfloat16())
    w = packing.dequant(q, s).double()
    assert np.array_equal(got, (w[:, 1:] @ x[1:].double()).numpy().astype(np.float32))


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_non_finite_activations_reach_every_row(bad):
    q, s, z = _matrix(300, 2560, True, 5)
    x = torch.randn(2560, generator=torch.Generator().manual_seed(6)).bfloat16()
    x[777] = bad
    assert not np.isfinite(_gemv(q, s, z, x)).any()
