"""Results brought to the host together (host side, with stand-in tensors)."""
import numpy as np
import torch

from sseqs_b200 import _lib


class _OnGpu(torch.Tensor):
    """A CPU tensor that says it is on a GPU."""
    is_cuda = property(lambda self: True)
    device = property(lambda self: self.where)


def _on(where, values):
    t = torch.tensor(values).as_subclass(_OnGpu)
    t.where = torch.device(where)
    return t


def test_every_device_with_a_result_is_waited_for(monkeypatch):
    """The copies are queued on the current stream of each tensor's device, so
    each of these streams is waited for, once and after its copies."""
    log = []
    empty = torch.empty

    def pinned(*args, pin_memory=False, **kw):
        assert pin_memory
        log.append("copy")
        return empty(*args, **kw)

    class Stream:
        def __init__(self, dev):
            self.dev = dev

        def synchronize(self):
            log.append(str(self.dev))

    monkeypatch.setattr(torch, "empty", pinned)
    monkeypatch.setattr(torch.cuda, "current_stream", Stream)
    src = [_on("cuda:0", [1, 2]), _on("cuda:1", [3]), _on("cuda:0", [4, 5, 6]), _on("cuda:1", [7])]
    out = _lib.to_host_many(src)
    assert log[:4] == ["copy"] * 4
    assert sorted(log[4:]) == ["cuda:0", "cuda:1"]
    for o, w in zip(out, ([1, 2], [3], [4, 5, 6], [7])):
        np.testing.assert_array_equal(o, w)
