"""What the multi-stage attention class refuses before the library is called, with a library that only takes notes: the
addresses of a batch element's parts are worked out by arithmetic, and nothing behind it looks at them again."""
import pytest
import torch

from infllm_b200 import _lib
from infllm_b200.attention import get_multi_stage_dot_production_attention


class _Notes:
    """Stands in for the library: no scratch, every call succeeds."""

    def __init__(self):
        self.calls = []

    def infllm_attn_stage_scratch(self, *args):
        return 0

    def infllm_attn_stage_ex(self, *args):
        self.calls.append(args)
        return 0

    infllm_attn_colsum = infllm_attn_stage_ex


@pytest.fixture
def notes(monkeypatch):
    n = _Notes()
    monkeypatch.setattr(_lib, "lib", n)
    monkeypatch.setattr(_lib, "require_cuda", lambda t, what: None)
    return n


def _rand(b, h, n):
    return torch.randn(b, h, n, 128).to(torch.bfloat16)


@pytest.mark.parametrize("kb,vb", [(1, 2), (2, 1), (1, 1), (0, 2)])
@pytest.mark.parametrize("get_score", [False, True])
def test_fewer_batch_elements_than_queries_have_are_refused(notes, monkeypatch, kb, vb, get_score):
    monkeypatch.setattr(_lib, "raw_stream", lambda device: 0)
    q = _rand(2, 4, 5)
    att = get_multi_stage_dot_production_attention(True)[0](q.shape, q.dtype, "cpu")
    with pytest.raises(IndexError):
        att.append(q, _rand(kb, 2, 9), _rand(vb, 2, 9), end=True, get_score=get_score)
    assert not notes.calls


@pytest.mark.parametrize("kb", [2, 3])
def test_as_many_or_more_are_taken(notes, monkeypatch, kb):
    monkeypatch.setattr(_lib, "raw_stream", lambda device: 0)
    q, k, v = _rand(2, 4, 5), _rand(kb, 2, 9), _rand(kb, 2, 9)
    att = get_multi_stage_dot_production_attention(True)[0](q.shape, q.dtype, "cpu")
    att.append(q, k, v, end=True, get_score=True)
    stage, sums = notes.calls[:2], notes.calls[2:]
    assert [(c[0], c[3], c[6]) for c in stage] == [(q[i].data_ptr(), k[i].data_ptr(), v[i].data_ptr()) for i in range(2)]
    assert [(c[0], c[3]) for c in sums] == [(q[i].data_ptr(), k[i].data_ptr()) for i in range(2)]


def test_a_stage_without_keys_has_no_batch_to_look_at(notes, monkeypatch):
    monkeypatch.setattr(_lib, "raw_stream", lambda device: 0)
    q = _rand(2, 4, 5)
    att = get_multi_stage_dot_production_attention(True)[0](q.shape, q.dtype, "cpu")
    att.append(q, _rand(1, 2, 0), _rand(1, 2, 0), end=True)
    assert len(notes.calls) == 2


def test_a_class_made_for_another_device_than_cuda_is_refused(notes, monkeypatch):
    # (a CUDA device that is there, so that only the class's own device is left to object to)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: 0, raising=False)
    q = _rand(1, 4, 5)
    att = get_multi_stage_dot_production_attention(True)[0](q.shape, q.dtype, "cpu")
    with pytest.raises(ValueError, match="cpu"):
        att.append(q, _rand(1, 2, 9), _rand(1, 2, 9), end=True)
    assert not notes.calls
    assert _lib.raw_stream(torch.device("cuda")) == _lib.raw_stream(torch.device("cuda:0")) == 0
