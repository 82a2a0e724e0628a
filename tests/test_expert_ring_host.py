"""The ring through which the expert products fetch their weights, on the host: how stages, slots and requesting warps go
together at every length of row."""
import ctypes
import importlib

import pytest

hyb = importlib.import_module("litespark_inference_b200.torchless.hybrid")
kernel = importlib.import_module("litespark_inference_b200.torchless.kernel")


@pytest.mark.parametrize("K", [64, 2560, 4096, 5120, 6912, 8192, 12288, 16384, 20000, 24640])
def test_a_slot_is_filled_by_one_warp(K):
    """Before a refill the requesting warp tests the phase of the slot's release.  One bit of phase tells two successive
    uses apart only to a warp that knows of the use before: the warp of all uses of the slot."""
    fn = kernel.load_library(require_device=False).lspk_debug_expert_stage
    fn.argtypes, fn.restype = hyb.SIGNATURES["lspk_debug_expert_stage"]
    slot, producer = ctypes.c_int(), ctypes.c_int()
    seen, uses = {}, {}
    for q in range(200):
        assert fn(K, q, ctypes.byref(slot), ctypes.byref(producer)) == 0
        assert seen.setdefault(slot.value, producer.value) == producer.value, (q, slot.value)
        uses.setdefault(slot.value, []).append(q)
    n = len(uses)
    assert n >= 3 and sorted(uses) == list(range(n))
    assert all(u == list(range(s, 200, n)) for s, u in uses.items())      # in turn
    assert len(set(seen.values())) == min(n, 4)                           # every requesting warp has work
