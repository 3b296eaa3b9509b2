"""The stream handle that the calls pass on: the current stream's, by torch's quick entry where it exists and
by the public one where it does not."""
import torch

import supereight2_gb300 as se


def test_handle_of_the_current_stream(monkeypatch):
    class Stream:
        cuda_stream = 0x1234

    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: Stream)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 0x5000 + device, raising=False)
    assert se._stream(None).value == 0x5003
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream")
    assert se._stream(None).value == 0x1234
    assert se._stream(7).value == 7
