"""The stream a drop-in kernel call without a queue runs on: the current one, also
where torch lacks its direct lookup."""
import types

import pytest
import torch

from pyugks_b200 import kernel_program as kp


@pytest.mark.parametrize("missing", ["_get_device", "_get_raw_stream"])
def test_without_the_direct_lookup(monkeypatch, missing):
    monkeypatch.setattr(kp, missing, None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=1234))
    assert kp._stream_ptr(None) == 1234
    assert kp._stream_ptr(77) == 77
    assert kp._stream_ptr(types.SimpleNamespace(cuda_stream=5)) == 5


@pytest.mark.gpu
def test_both_lookups_agree(cuda, monkeypatch):
    for s in (torch.cuda.current_stream(), torch.cuda.Stream()):
        with torch.cuda.stream(s):
            assert kp._stream_ptr(None) == s.cuda_stream
            with monkeypatch.context() as m:
                m.setattr(kp, "_get_raw_stream", None)
                assert kp._stream_ptr(None) == s.cuda_stream
