"""Resuming paused memory that training passes have cached meanwhile (on the CPU, with a device that is counted)."""
import pytest
import torch

from miles_b200.utils.memory_saver import MemorySaver

GB = 1 << 30


class Device:
    """A device of 100 GB whose arena has 60 GB paused; the allocator's cache gives back what it holds."""

    def __init__(self, cached):
        self.mapped, self.cached, self.emptied = 0, cached, 0

    def free(self):
        return 100 * GB - self.mapped - self.cached

    def vmm_stats(self):
        return {"kv": (self.mapped, 60 * GB - self.mapped), "default": (0, 0)}

    def vmm_resume(self, tag):
        if self.free() < 60 * GB:
            raise RuntimeError("out of device memory while resuming tag " + tag)
        self.mapped = 60 * GB
        return self.mapped

    def empty_cache(self):
        self.cached, self.emptied = 0, self.emptied + 1


@pytest.mark.parametrize("cached, emptied", [(0, 0), (30, 0), (39, 0), (40, 1), (70, 1), (100, 1)])
def test_cached_memory_is_given_back_where_it_is_needed(monkeypatch, cached, emptied):
    dev = Device(cached * GB)
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (dev.free(), 100 * GB))
    monkeypatch.setattr(torch.cuda, "empty_cache", dev.empty_cache)
    saver = object.__new__(MemorySaver)
    saver.C, saver.available = dev, True
    assert saver.resume("kv") == 60 * GB and dev.emptied == emptied
