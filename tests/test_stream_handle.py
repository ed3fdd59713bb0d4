"""The stream handle passed to the library: torch's raw entry where the build has it, the public
Stream object otherwise.  CPU only, with stand-ins for both."""
import types

import torch


def test_public_stream_where_the_raw_entry_is_missing(monkeypatch):
    from mmnorm_b200 import ops
    seen = []

    def current(device):
        seen.append(device)
        return types.SimpleNamespace(cuda_stream=0x1230)

    monkeypatch.setattr(ops, "_raw_stream", None)
    monkeypatch.setattr(torch.cuda, "current_stream", current)
    assert ops._stream(torch.device("cuda", 1)).value == 0x1230
    assert seen == [torch.device("cuda", 1)]


def test_raw_entry_gets_the_device_index(monkeypatch):
    from mmnorm_b200 import ops
    monkeypatch.setattr(ops, "_raw_stream", lambda index: 0x40 + index)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 2)
    assert ops._stream(torch.device("cuda", 1)).value == 0x41
    assert ops._stream(torch.device("cuda")).value == 0x42
