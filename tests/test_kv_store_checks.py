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
    monkeypatch.setattr(kv_store, "_device", lambda: 3)
    monkeypatch.setattr(kv_store, "_stream", lambda device: 4096 + device)
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
        args["slot_mapping"].data_ptr(), n, 1024, kc.shape[0] * kc.shape[1], 0, 4099))])


@pytest.mark.parametrize("changed", [
    dict(value=rows(4)), dict(value=rows(5, 4)), dict(value=rows(5, dtype=torch.float16)), dict(value=rows(5, dtype=torch.float32)),
    dict(v_cache=cache(3)), dict(v_cache=cache(4, 32)), dict(v_cache=cache(dtype=torch.float16)),
    dict(k_cache=cache(8)[::2]), dict(v_cache=torch.zeros(4, 2, 64, 8, 128, dtype=BF)[:, 1]), dict(slot_mapping=ints(4)),
    dict(slot_mapping=ints(5, dtype=torch.int64)), dict(key=rows(5, dtype=torch.float16)), dict(k_cache=cache(dtype=torch.float16))])
def test_store_refuses(calls, changed):
    with pytest.raises((AssertionError, TypeError)):
        kv_store.store_kvcache(**store_args(**changed))
    assert not calls


def prefill_args(cached=False, **changed):
    q = torch.zeros(6, 16, 128, dtype=BF)
    kv = (cache(), cache()) if cached else (rows(6), rows(6))
    args = dict(q=q, k=kv[0], v=kv[1], cu_seqlens_q=ints(3), max_seqlen_q=4, softmax_scale=0.125)
    if cached:
        args.update(cu_seqlens_k=ints(3), block_table=ints(2, 5))
    args.update(changed)
    return args


@pytest.mark.parametrize("cached,changed", [
    (False, dict()), (False, dict(cu_seqlens_k=ints(3))), (False, dict(v=torch.zeros(6, 4096, dtype=BF)[:, 3072:].view(6, 8, 128))),
    (False, dict(k=rows(9))), (False, dict(v=rows(9))), (False, dict(v=rows(6, 16))), (False, dict(cu_seqlens_k=ints(7))),
    (False, dict(k=rows(6).view(6, 8, 2, 64), v=rows(6).view(6, 8, 1, 128))), (True, dict(k=cache().view(4, 64, 8, 2, 64))), (True, dict()), (True, dict(v=cache(6))),
    (True, dict(k=torch.zeros(2, 4, 64, 8, 128, dtype=BF)[0], block_table=ints(3, 8)[:, :2])),
    (True, dict(k=cache(1), v=torch.zeros(1, 2, 64, 8, 128, dtype=BF)[:, 0]))])
def test_prefill_takes(calls, cached, changed):
    a = prefill_args(cached, **changed)
    out = kv_store.prefill_attention(**a)
    k, v, cu_k, table = a["k"], a["v"], a.get("cu_seqlens_k"), a.get("block_table")
    assert tuple(out.shape) == (6, 16, 128) and out.dtype == BF
    assert calls == [("_prefill", (
        a["q"].data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), a["cu_seqlens_q"].data_ptr(),
        0 if cu_k is None else cu_k.data_ptr(), 2, 4, 2048, k.stride(int(cached)), v.stride(int(cached)), 2048, 16, 8, 128, 0.125,
        table.data_ptr() if cached else 0, table.stride(0) if cached else 0, 64 if cached else 0, len(k) if cached else 0, 0, 6,
        0 if cached else min(len(k), len(v)), 4099))]


@pytest.mark.parametrize("cached,changed", [
    (False, dict(v=rows(6, 4))), (False, dict(cu_seqlens_k=ints(3, dtype=torch.int64))), (False, dict(cu_seqlens_k=ints(2))),
    (False, dict(cu_seqlens_k=torch.zeros(3, dtype=torch.int32))), (False, dict(v=torch.zeros(6, 8, 256, dtype=BF)[:, :, :128])),
    (False, dict(k=rows(6)[:, :, :64])), (False, dict(v=rows(6, dtype=torch.float16))), (False, dict(cu_seqlens_q=ints(3, dtype=torch.int64))),
    (True, dict(v=cache(3))), (True, dict(v=cache(8, 32))), (True, dict(v=torch.zeros(4, 2, 64, 8, 128, dtype=BF)[:, 1])),
    (True, dict(k=cache(8)[::2])), (True, dict(v=cache(heads=4))), (True, dict(cu_seqlens_k=ints(3, dtype=torch.int64))),
    (True, dict(cu_seqlens_k=ints(2))), (True, dict(cu_seqlens_k=None)), (True, dict(block_table=torch.zeros(2, 5, dtype=torch.int32))),
    (True, dict(block_table=ints(2, 5, dtype=torch.int64))), (True, dict(block_table=ints(1, 5)))])
def test_prefill_refuses(calls, cached, changed):
    with pytest.raises((AssertionError, TypeError)):
        kv_store.prefill_attention(**prefill_args(cached, **changed))
    assert not calls
