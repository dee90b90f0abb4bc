"""Which devices a blocking status check waits for, and what it raises, with the native path and CUDA replaced by stand-ins."""
import pytest
import torch

from swamla_b200 import _cabi, functional, status


class Native:
    def __init__(self, devices, error=None):
        self.devices, self.error, self.polled = devices, error, 0

    def devices_used(self):
        return self.devices

    def poll_status(self):
        self.polled += 1
        if self.error:
            raise _cabi.LmoeError(self.error)


class Event:
    def __init__(self):
        self.waited = False

    def synchronize(self):
        self.waited = True

    def query(self):
        return True


@pytest.fixture
def cuda(monkeypatch):
    """The devices that were synchronised; ``cuda.capturing`` answers for the current stream."""
    class Cuda:
        synced, capturing = [], False
    c = Cuda()
    c.synced = []
    monkeypatch.setattr(torch.cuda, "synchronize", lambda d=None: c.synced.append(d))
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: c.capturing)
    monkeypatch.setattr(status, "_pending", [])
    return c


def test_every_used_device_is_waited_for(cuda, monkeypatch):
    native = Native([0, 3])
    monkeypatch.setattr(functional, "_native", native)
    status.poll(block=True)
    assert cuda.synced == [0, 3] and native.polled == 1


def test_nothing_is_waited_for_while_capturing_or_before_any_step(cuda, monkeypatch):
    monkeypatch.setattr(functional, "_native", Native([0]))
    cuda.capturing = True
    status.poll(block=True)
    assert cuda.synced == []
    monkeypatch.undo()
    monkeypatch.setattr(functional, "_native", None)
    status.poll(block=True)                  # on a machine without a GPU too


def test_pending_steps_are_looked_at_before_a_failure_is_raised(cuda, monkeypatch):
    monkeypatch.setattr(functional, "_native", Native([1], "device status 101 in LatentMoE forward on cuda:1"))
    ev, word = Event(), torch.zeros(1, dtype=torch.int32)
    monkeypatch.setattr(status, "_pending", [(ev, word, "expert-parallel step")])
    with pytest.raises(_cabi.LmoeError, match="cuda:1"):
        status.poll(block=True)
    assert ev.waited and status.pending() == 0
    status._free.remove(word)
