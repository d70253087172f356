"""What ``store_kvcache`` and ``prefill_attention`` hand to the library, and what they refuse: tensors that the kernels would
read or write beyond, or at other places than the views say.  No GPU work: the native calls are replaced by a recorder."""

import struct

import pytest
import torch

from dfb_b200 import kv_store

BF = torch.bfloat16


class OnDevice(torch.Tensor):
    """A tensor that says that it lies on the GPU."""
    is_cuda = True


@pytest.fixture
def calls(monkeypatch):
    kv_store._load()
    seen = []
    for name, form in (("_store", "12q"), ("_prefill", "15qd8q")):
        monkeypatch.setattr(kv_store, name, lambda words, name=name, form=form: seen.append((name, struct.unpack(form, words))) and 0)
    monkeypatch.setattr(kv_store, "_stream", lambda: 0)
    return seen


def rows(n, heads=8, dim=128, dtype=BF):
    return torch.zeros(n, heads, dim, dtype=dtype)


def cache(blocks=4, size=64, heads=8, dtype=BF):
    return torch.zeros(blocks, size, heads, 128, dtype=dtype)


def ints(*shape, dtype=torch.int32):
    return torch.zeros(*shape, dtype=dtype).as_subclass(OnDevice)


def store_args(**changed):
    args = dict(key=rows(5), value=rows(5), k_cache=cache(), v_cache=cache(), slot_mapping=ints(5))
    args.update(changed)
    return args


@pytest.mark.parametrize("changed", [
    dict(), dict(value=torch.zeros(5, 4096, dtype=BF)[:, 3072:].view(5, 8, 128)), dict(value=rows(9)),
    dict(k_cache=cache().flatten(2), v_cache=cache().flatten(2)), dict(k_cache=cache().flatten(2)), dict(v_cache=cache(6)),
    dict(k_cache=cache(8)[2:6], v_cache=torch.zeros(2, 4, 64, 8, 128, dtype=BF)[1]),
    dict(k_cache=torch.zeros(1, 2, 64, 8, 128, dtype=BF)[:, 0], v_cache=cache(1)),         # one block: no step to the next
    dict(k_cache=cache(2, 128)), dict(key=rows(0), value=rows(0), slot_mapping=ints(0))])
def test_store_takes(calls, changed):
    args = store_args(**changed)
    kv_store.store_kvcache(**args)
    n, kc = len(args["key"]), args["k_cache"]
    assert [c for c in calls] == ([] if n == 0 else [("_store", (
        args["key"].data_ptr(), args["value"].data_ptr(), 1024, args["value"].stride(0), kc.data_ptr(), args["v_cache"].data_ptr(),
        args["slot_mapping"].data_ptr(), n, 1024, kc.shape[0] * kc.shape[1], 0, 0))])


@pytest.mark.parametrize("changed", [
    dict(value=rows(4)), dict(value=rows(5, 4)), dict(value=rows(5, dtype=torch.float16)), dict(value=rows(5, dtype=torch.float32)),
    dict(v_cache=cache(3)), dict(v_cache=cache(4, 32)), dict(v_cache=cache(dtype=torch.float16)),
    dict(k_cache=cache(8)[::2]), dict(v_cache=torch.zeros(4, 2, 64, 8, 128, dtype=BF)[:, 1]), dict(slot_mapping=ints(4)),
    dict(slot_mapping=ints(5, dtype=torch.int64)), dict(key=rows(5, dtype=torch.float16)), dict(k_cache=cache(dtype=torch.float16))])
def test_store_refuses(calls, changed):
    with pytest.raises((AssertionError, TypeError)):
        kv_store.store_kvcache(**store_args(**changed))
    assert not calls
