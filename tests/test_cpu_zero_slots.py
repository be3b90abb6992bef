"""Slot numbers outside of the state storage are refused on the host, before the kernel that zeroes them writes anywhere."""
import pytest
import torch


@pytest.mark.parametrize("slots", [[8], [0, 3, 8], [-9], [1 << 40]])
def test_slots_outside_of_the_storage_are_refused(slots, monkeypatch):
    from llm_b200.csrc import ops
    monkeypatch.setattr(ops, "load", lambda: pytest.fail("a launch"))
    with pytest.raises(IndexError):
        ops.zero_slots(torch.zeros(2, 2, dtype=torch.int64), 64, slots, 8)


def test_the_storage_tells_how_many_slots_it_has(monkeypatch):
    from llm_b200.cache.storage import StateStorage
    from llm_b200.csrc import ops
    from llm_b200.parts.base import StateNeed
    store = StateStorage([StateNeed((4,)), StateNeed((3, 2))], 8, torch.device("cpu"))
    told = []
    monkeypatch.setattr(ops, "zero_slots", lambda regions, most, slots, held: told.append((most, slots, held)))

    class OnDevice:
        is_cuda = True
    store._regions = OnDevice()
    store.zero_slots([7, -8])
    assert told == [(24, [7, -8], 8)]
