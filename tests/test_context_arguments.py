"""CPU checks of how the Python layer finds a context and a stream, with the library's calls
and torch's CUDA state replaced by fakes."""
import types

import numpy as np


class FakeLib:
    def __init__(self):
        self.bound = []

    def qed2d_ctx_create(self, L1, L2, beta, out):
        out._obj.value = 1000 * L1 + L2
        return 0

    def qed2d_ctx_set_precision(self, h, p):
        return 0

    def qed2d_ctx_bind(self, h, beta, stream):
        self.bound.append((h, beta, stream))
        return 0


def test_context_extents_and_stream(monkeypatch):
    import torch
    import qed2d
    fake = FakeLib()
    monkeypatch.setattr(qed2d, "lib", lambda: fake)
    monkeypatch.setattr(qed2d, "_ctx", {})
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: types.SimpleNamespace(cuda_stream=77))
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda dev: 55, raising=False)
    # whatever int() takes as an extent: one context
    for L1, L2 in ((6, 4), (np.int64(6), 4.0), (np.array(6), np.array(4)), (torch.tensor(6), 4), ("6", "4")):
        assert qed2d.context(L1, L2, 2.0) == 6004
    assert len(qed2d._ctx) == 1 and set(fake.bound) == {(6004, 2.0, 55)}
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream")
    qed2d.context(6, 4, 2.0)
    assert fake.bound[-1] == (6004, 2.0, 77)
