"""The stream of calls without one: torch's current one, also with a torch that lacks the calls it is asked for directly with."""
import sys

import pytest

from __graft_entry__ import load_package


@pytest.mark.parametrize("missing", [(), ("_cuda_getCurrentRawStream",), ("_cuda_getDevice",)])
@pytest.mark.parametrize("initialised", [False, True])
def test_the_stream_of_a_call_without_one(monkeypatch, missing, initialised):
    import torch

    load_package()
    pkg = "cccc_lite_b200."
    monkeypatch.setattr(torch.cuda, "is_initialized", lambda: initialised)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: type("Stream", (), dict(cuda_stream=77))())
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 3, raising=False)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 1000 + device, raising=False)
    for name in missing:
        monkeypatch.delattr(torch._C, name)
    want = 1003 if initialised and not missing else 77
    assert sys.modules[pkg + "torch_stream"].raw_stream() == want
    capi = sys.modules[pkg + "capi"]
    assert capi._stream(None) == want and capi._stream(0) == 0 and capi._stream(5) == 5
