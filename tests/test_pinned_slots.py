"""Pinned buffers and their events around the native copies of a step, with a fake CUDA (no GPU)."""
import pytest
import torch

from minfer_b200.kernels import api as K


class FakeStream:
    cuda_stream = 7


class FakeCuda:
    """Keeps the device that is current, and which device an event's handle was made on."""

    def __init__(self):
        self.device, self.made_on, self.calls, self.waits = 0, {}, [], []
        cuda = self

        class Event:
            cuda_event = 0

            def record(self):
                if not self.cuda_event:
                    self.cuda_event = len(cuda.made_on) + 1
                    cuda.made_on[self.cuda_event] = cuda.device

            def synchronize(self):
                pass

        self.Event = Event

    def launcher(self, name, events):
        def call(*args):
            self.calls.append((name, [self.made_on[args[i]] for i in events if args[i] is not None]))
            return 0
        return call


@pytest.fixture
def cuda(monkeypatch):
    fake = FakeCuda()
    fake.mf_step_inputs = fake.launcher("step_inputs", [5])
    fake.mf_copy_back = fake.launcher("copy_back", [3, 4])
    fake.mf_event_wait = lambda handle: fake.waits.append(handle)
    monkeypatch.setattr(torch.cuda, "Event", fake.Event)
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda self: self)
    monkeypatch.setattr(K, "_lib", lambda name: fake)
    monkeypatch.setattr(K, "_ptr", lambda t, what="tensor": None if t is None else t.data_ptr())
    monkeypatch.setattr(K, "_stream", lambda: 0)
    return fake


def test_a_slot_made_while_another_device_is_current_can_be_used(cuda):
    """An event belongs to the device that was current when its handle was made, and only streams of that
    device can record it: the copies' device counts, not the one where the slot was made."""
    slot = K.PinnedSlot(4)
    cuda.device = 1
    dev = torch.zeros(4, dtype=torch.int32)
    K.copy_back(slot, dev)
    K.copy_back(slot, dev, FakeStream())
    K.step_inputs(dev, slot, None)
    assert cuda.calls == [("copy_back", [1]), ("copy_back", [1, 1]), ("step_inputs", [1])]


def test_a_slot_that_goes_waits_for_a_copy_that_nobody_has_waited_for(cuda):
    dev = torch.zeros(4, dtype=torch.int32)
    for copies, waited in ((0, False), (1, False), (2, True), (1, True)):
        cuda.waits.clear()
        slot = K.PinnedSlot(4)
        for _ in range(copies):
            K.copy_back(slot, dev)
        if waited:
            slot.wait()
        handle = slot.handle
        del slot
        assert cuda.waits == ([handle] if copies and not waited else [])
