"""Entry points called with plain lists of tensors where they take arrays of
pointers (host only: the native call is replaced)."""
import ctypes
import weakref

import pytest
import torch


@pytest.mark.parametrize("entry", ["convert_correct_tiles", "process_frame"])
def test_arrays_of_lists_live_through_the_call(monkeypatch, entry):
    """Every array made from a list is there, with its own list's addresses,
    when the native function is called."""
    from tile_processor_gpu_b200 import _native, api
    made = []

    class Array(api.PointerArray):
        def __init__(self, tensors, device=None):
            super().__init__(tensors, device)
            made.append((weakref.ref(self.dev), [t.data_ptr() for t in tensors]))

    lists = [[torch.zeros(4) for _ in range(4)] for _ in range(4)]
    addresses = [[t.data_ptr() for t in x] for x in lists]
    calls = []

    def call(name, *args):
        assert len(made) == 4
        for ref, want in made:
            dev = ref()
            assert dev is not None and dev.tolist() == want
        at = {tuple(want): ref().data_ptr() for ref, want in made}
        for a, want in zip(args[1:4], addresses):
            ctypes.c_void_p.from_param(a)
            assert a._as_parameter_.value == at[tuple(want)]
        calls.append(name)
        return 0

    monkeypatch.setattr(api, "PointerArray", Array)
    monkeypatch.setattr(_native, "call", call)
    g = api.Geometry(64, 64)
    t, x = torch.zeros((4, 10), dtype=torch.int32), torch.zeros(8)
    if entry == "convert_correct_tiles":
        api.convert_correct_tiles(g, *lists[:3], t, lists[3], 64, 4)
    else:
        api.process_frame(g, *lists[:3], 64, t, 4, x, 225, x, t, t, t, 72, x, gpu_clt=lists[3])
    assert len(calls) == 1
