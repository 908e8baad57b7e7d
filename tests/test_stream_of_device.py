"""CPU: tensors that are not on a GPU are refused before the library sees their pointers."""
import ctypes

import pytest
import torch

from flint_b200 import draft, engine
from flint_b200.draft import DraftHead


class _Library:
    """Stands in for the C library: a launch is a failure of the test."""

    def __getattr__(self, name):
        def call(*args):
            raise AssertionError(f"{name} called")
        return call

    def fb_draft_destroy(self, handle):
        return 0


@pytest.fixture
def head():
    m = DraftHead(512, 8, 256)
    m.lib, m._h = _Library(), ctypes.c_void_p(1)
    yield m
    m.close()


def test_draft_forward_refuses_features_on_the_cpu(head):
    with pytest.raises(ValueError, match="cuda device"):
        head(torch.zeros(2, 512, dtype=torch.bfloat16), tokens=torch.zeros(2, dtype=torch.int32))


def test_draft_forward_refuses_embeddings_on_the_cpu(head, monkeypatch):
    monkeypatch.setattr(draft, "_stream_ptr", lambda device: 0)          # as if the features were where they should be
    with pytest.raises(ValueError, match="emb"):
        head(torch.zeros(2, 512, dtype=torch.bfloat16), torch.zeros(2, 512, dtype=torch.bfloat16))


def test_draft_head_refuses_rows_on_the_cpu(head):
    with pytest.raises(ValueError, match="cuda device"):
        head.head(torch.zeros(1, 512, dtype=torch.bfloat16))


def test_stream_is_the_device_s_own(monkeypatch):
    seen = []
    monkeypatch.setattr(engine, "_raw_stream", lambda index: seen.append(index) or 77)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    assert engine._stream_ptr(torch.device("cuda:1")) == 77 and engine._stream_ptr(torch.device("cuda")) == 77
    assert seen == [1, 3]
    with pytest.raises(ValueError):
        engine._stream_ptr(torch.device("cpu"))
