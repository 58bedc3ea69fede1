"""The launches with which a request takes its slot: zeros in the slot of every state array, and its sampling constants and
generator state."""
import types

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cache(max_sequences, shapes):
    from cuca_b200.cache.device import DeviceCache
    from cuca_b200.parts.base import CacheNeeds, StateNeeds
    rt = types.SimpleNamespace(device=torch.device("cuda:0"), dtype=torch.float32)
    needs = {i: CacheNeeds(state=StateNeeds(*s) if isinstance(s, tuple) else {n: StateNeeds(*v) for n, v in s.items()})
             for i, s in enumerate(shapes)}
    return DeviceCache(rt, [], 16, needs, max_sequences, 64)


SHAPES = [((5,), "int32"), ((3, 7), "float32"), {"a": ((16, 4),), "b": ((3,), "bfloat16")}, ((1,), "bfloat16"),
          ((130, 33), "float32"), ((256, 256), "float32")]


@pytest.mark.parametrize("max_sequences", [1, 2, 9])
def test_a_slot_is_cleared_and_no_other(max_sequences):
    """State arrays whose slots are 2 to 262,144 bytes, most of them not of 16-byte multiples: first, middle and last slot,
    counted from either end; every other byte stays. The same after arrays were replaced, one by a strided view."""
    cache = _cache(max_sequences, SHAPES)

    def check(slot):
        before = []
        for t in cache._state_tensors():
            g = torch.Generator(device=t.device).manual_seed(t.numel() + slot % 7)
            t.copy_(torch.randint(1, 100, t.shape, device=t.device, generator=g))
            before.append(t.clone())
        cache.clear_slot(slot)
        for t, b in zip(cache._state_tensors(), before):
            b[slot] = 0
            assert torch.equal(t, b), (slot, tuple(t.shape))

    slots = sorted({0, max_sequences // 2, max_sequences - 1, -1, -max_sequences})
    for slot in slots:
        check(slot)
    cache.state[1] = torch.empty_like(cache.state[1])
    check(max_sequences - 1)
    cache.state[1] = torch.empty(max_sequences, 5, 7, device="cuda:0")[:, 1:4]  # slots lie further apart than their bytes
    check(max_sequences - 1)
    cache.state[4] = torch.empty(max_sequences, 33, 130, device="cuda:0").transpose(1, 2)
    check(max_sequences // 2)
    for slot in (max_sequences, -max_sequences - 1):
        with pytest.raises(IndexError):
            cache.clear_slot(slot)


@pytest.mark.parametrize("state", [0, 1, (1 << 63) - 1, 1 << 63, (1 << 64) - 1])
@pytest.mark.parametrize("slot", [0, 3, 6])
def test_a_slots_sampling_constants_arrive(state, slot):
    from cuca_b200.kernels import ops
    dev = torch.device("cuda:0")
    rng = torch.full((7,), -5, dtype=torch.int64, device=dev)
    temperature, top_p = torch.full((7,), 9.0, device=dev), torch.full((7,), 8.0, device=dev)
    top_k = torch.full((7,), 4, dtype=torch.int32, device=dev)
    ops.set_sampling(rng, temperature, top_k, top_p, slot, state, 0.7, (1 << 31) - 1, 0.95)
    want = [-5] * 7
    want[slot] = state - (1 << 64) if state >> 63 else state
    assert rng.tolist() == want
    for got, value, rest in ((temperature, np.float32(0.7), 9.0), (top_p, np.float32(0.95), 8.0), (top_k, (1 << 31) - 1, 4)):
        assert got.tolist() == [value if i == slot else rest for i in range(7)]
    for bad in (-1, 7):
        with pytest.raises(IndexError):
            ops.set_sampling(rng, temperature, top_k, top_p, bad, 1, 1.0, 1, 1.0)
    with pytest.raises(OverflowError):
        ops.set_sampling(rng, temperature, top_k, top_p, 0, 1, 1.0, 1 << 31, 1.0)
