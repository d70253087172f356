"""Steps of 9 to 32 slots in one pass over the weights (``dfb_wide.cuh``) against the same step taken in launches of 8
rows (DFB_OPT_SLOTS_WIDE = 0): one, several and all rows of the last group of 8, contexts of one token, around
chunk and block boundaries and of the full model length, sampled rows in some groups (the noise stream is the one of the
launches of 8).  One step from the same state: the new cache rows and the tokens.  Also against the fp32 oracle, as a
serving loop, with an error status, with options, without room for its buffers."""

import numpy as np
import pytest
import torch

from oracle import qwen3_decode as O
from tests import harness as H

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
LENGTHS = [40, 0, 255, 1300, 64, 512, 901, 17, 63, 128, 1020, 256, 450, 600, 5, 2046, 860, 1500, 390, 95, 1, 777, 1023,
           33, 2, 65, 127, 1800, 300, 71, 700, 192]


@pytest.fixture(scope="module")
def model():
    g = H.oracle_geometry(layers=2, vocab=4096)
    w = O.make_weights(g, seed=91, norm="random").to(BF)
    # a clear winner for every row: even and odd rows of the embedding are images under the final norm's signs
    signs = torch.from_numpy(np.random.Generator(np.random.Philox(key=93)).integers(0, 2, g.hidden)).to(BF) * 2 - 1
    w.embed.copy_(torch.randn(g.vocab, g.hidden, generator=torch.Generator().manual_seed(94)) * 0.5)
    w.embed[1::2] = w.embed[0::2] * signs
    w.final_norm.copy_(signs)
    blocks = sum((n + 1) // 256 + 1 for n in LENGTHS)
    history = torch.from_numpy(np.random.Generator(np.random.Philox(key=92)).standard_normal(
        tuple(O.new_kv_cache(g, blocks, BF).shape), dtype=np.float32) * 0.5).to(BF).cuda()
    return g, w, history


def _step(w, history, n, temperatures, wide, steps=1, use_graph=True, before_steps=None):
    from dfb_b200 import native
    from dfb_b200.slots import SlotRuntime
    kv = history.clone()
    dec = H.make_decoder(w, kv, use_graph=use_graph)
    if not wide:
        dec.set_option(native.DFB_OPT_SLOTS_WIDE, 0)
    dec.set_seed(5)
    rt = SlotRuntime(dec)
    first = 0
    for i in range(n):
        blocks = (LENGTHS[i] + steps - 1) // 256 + 1
        rt.admit(i, 100 + 7 * i, LENGTHS[i], list(range(first, first + blocks)), temperatures[i] if temperatures else 0.0)
        first += blocks
    if before_steps:
        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.default_stream()):
            before_steps()
    out = [rt.step() for _ in range(steps)]
    assert dec.status()[0] == 0
    dec.close()
    return out, kv


@pytest.mark.parametrize("n", [9, 16, 17, 23, 25, 32])
@pytest.mark.parametrize("sampled", [False, True])
def test_wide_step_equals_steps_of_eight(model, cuda_device, n, sampled):
    g, w, history = model
    # groups 0 and 2 have sampled rows, group 1 none: only sampled groups advance the noise stream
    temps = [0.7 if sampled and i // 8 != 1 and i % 3 == 0 else 0.0 for i in range(n)]
    got, kv_got = _step(w, history, n, temps, wide=True)
    want, kv_want = _step(w, history, n, temps, wide=False)
    diff = (kv_got.float() - kv_want.float()).abs().max()
    assert float(diff) <= 2.0 ** -5, float(diff)
    changed = (kv_got != history).any(dim=-1)
    assert torch.equal(changed, (kv_want != history).any(dim=-1))          # exactly the same slots were written
    assert got[0] == want[0]


def test_wide_step_noise_stream_continues(model, cuda_device):
    """Two steps: the second one's noise starts where the first one's groups left the counter."""
    g, w, history = model
    temps = [5.0] * 20
    got, _ = _step(w, history, 20, temps, wide=True, steps=1)
    more, _ = _step(w, history, 20, temps, wide=True, steps=2)
    want, _ = _step(w, history, 20, temps, wide=False, steps=2)
    assert more[0] == got[0] and more[1] != more[0]
    assert sum(more[1][i] == want[1][i] for i in range(20)) >= 18          # (a near tie may fall the other way)


def test_first_wide_step_beside_a_busy_default_stream(model, cuda_device):
    """The buffers of a wide step are made by the first one: they are ready for a step on a stream of its own, whatever
    the default stream is still doing (30 products of 8,192 x 8,192 matrices, several ms)."""
    g, w, history = model
    want, kv_want = _step(w, history, 12, None, wide=True)
    a = torch.zeros(8192, 8192, dtype=BF, device="cuda")
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        got, kv_got = _step(w, history, 12, None, wide=True, use_graph=False,
                            before_steps=lambda: [torch.mm(a, a) for _ in range(30)])
    torch.cuda.synchronize()
    assert got == want and torch.equal(kv_got, kv_want)


def _held(dec):
    """Graphs that the decoder holds (of a refused call, which prepares nothing)."""
    import ctypes as C
    n = C.c_int32(0)
    assert dec._lib.dfb_warm(dec._handle, 0, 1, 1, C.byref(n)) == -1
    return n.value


def _tables(n, lengths):
    first = np.cumsum([0] + [lengths[i] // 256 + 2 for i in range(n)])
    return [list(range(first[i], first[i + 1])) for i in range(n)], int(first[-1])


@pytest.mark.parametrize("sampled", [False, True])
def test_serving_on_the_default_kernels(model, cuda_device, sampled):
    """Sequences that join, retire, change slots and wait for a block, with 6 to 20 live slots (8 and 9 among them), on the
    kernels that a user gets, step for step beside a decoder that takes launches of 8.  The steps capture and
    allocate nothing."""
    from dfb_b200 import native
    from dfb_b200.slots import SlotRuntime
    g, w, _ = model
    n_seq = 26
    rng = np.random.Generator(np.random.Philox(key=95))
    lens = [int(x) for x in rng.integers(1, 1400, n_seq)]
    lens[2], lens[5] = 255, 511                                        # run out of their first blocks after one token
    tables, blocks = _tables(n_seq, lens)
    budget = [int(x) for x in rng.integers(3, 16, n_seq)]
    temps = [4.0 if sampled and i % 5 == 0 else 0.0 for i in range(n_seq)]
    history = torch.from_numpy(rng.standard_normal(tuple(O.new_kv_cache(g, blocks, BF).shape), dtype=np.float32) * 0.5).to(BF).cuda()
    kinds = dict(kinds=8 | 16 | 32)                                    # host buffers, sampling; the slots' by the runtime
    sides = []
    for wide in (True, False):
        kv = history.clone()
        dec = H.make_decoder(w, kv)
        if not wide:
            dec.set_option(native.DFB_OPT_SLOTS_WIDE, 0)
        dec.set_seed(11)
        dec.warm(**kinds)
        sides.append((SlotRuntime(dec), dec, kv))
    held, free = _held(sides[0][1]), None
    assert held > _held(sides[1][1])                                   # the wide steps' graphs are there
    slot_of, order, left = {}, list(range(n_seq)), dict(enumerate(budget))
    free_slots = [int(x) for x in rng.permutation(32)]
    seen, misses, draws, waited = set(), 0, 0, set()

    def admit(i):
        slot_of[i] = free_slots.pop(0)
        for rt, _, _ in sides:
            rt.admit(slot_of[i], 100 + 7 * i, lens[i], tables[i][:lens[i] // 256 + 1], temps[i])

    targets = [20, 20, 18, 9, 8, 9, 6, 12, 20, 17, 16, 9, 8, 7, 6, 5, 4, 3]
    for step in range(200):
        while order and len(slot_of) < targets[min(step, len(targets) - 1)]:
            admit(order.pop(0))
        if not slot_of:
            break
        a, b = sides[0][0].step(), sides[1][0].step()
        if step == 1:
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
        assert set(a) == set(b)
        seen.add(len(a))
        for i, slot in list(slot_of.items()):
            if slot not in a:                                          # waits for its next block
                waited.add(i)
                for rt, _, _ in sides:
                    rt.extend(slot, tables[i])
                continue
            if temps[i]:
                draws += 1
                if a[slot] != b[slot]:                                 # a near tie: both go on with the same token
                    misses += 1
                    _, _, pos = sides[1][0].state(slot)
                    sides[1][0].admit(slot, a[slot], pos, tables[i][:pos // 256 + 1], temps[i])
            else:
                assert a[slot] == b[slot], (step, i)
            left[i] -= 1
            if left[i] == 0 or (step in (3, 5) and len(slot_of) > targets[step + 1]):
                for rt, _, _ in sides:
                    rt.retire(slot)
                free_slots.append(slot_of.pop(i))
    assert not order and waited >= {2, 5} and {8, 9} <= seen and max(seen) == 20, (seen, waited)
    assert misses <= draws // 20, (misses, draws)
    assert _held(sides[0][1]) == held
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free
    kv_a, kv_b = sides[0][2], sides[1][2]
    assert torch.equal((kv_a != history).any(-1), (kv_b != history).any(-1))
    assert float((kv_a.float() - kv_b.float()).abs().max()) <= 2.0 ** -5
    for _, dec, _ in sides:
        assert dec.status()[0] == 0
        dec.close()


def test_warm_prepares_the_wide_steps(model, cuda_device):
    """``dfb_warm`` of the host-buffer steps of 8 rows covers the slots' steps whatever their number, as it says."""
    from dfb_b200.slots import SlotRuntime
    g, w, history = model
    dec = H.make_decoder(w, history.clone())
    held = dec.warm(kinds=dec.WARM_HOST | dec.WARM_SAMPLING)
    assert held == _held(dec)
    rt = SlotRuntime(dec)
    first = 0
    for i in range(32):
        rt.admit(i, 100 + 7 * i, LENGTHS[i], list(range(first, first + LENGTHS[i] // 256 + 1)), 0.5 if i % 4 == 0 else 0.0)
        first += LENGTHS[i] // 256 + 1
        if i >= 8:
            rt.step()
            for j in range(i + 1):                                      # the same position again
                rt.admit(j, 100 + 7 * j, LENGTHS[j], list(range(sum(n // 256 + 1 for n in LENGTHS[:j]),
                                                                sum(n // 256 + 1 for n in LENGTHS[:j + 1]))), 0.5 if j % 4 == 0 else 0.0)
    assert _held(dec) == held
    dec.close()


def test_no_room_for_the_wide_buffers(model, cuda_device):
    """A decoder whose memory went to the cache before the first step of more than 8 slots takes launches of 8."""
    from dfb_b200.slots import SlotRuntime
    g, w, history = model
    want, kv_want = _step(w, history, 12, None, wide=False)
    kv = history.clone()
    dec = H.make_decoder(w, kv)
    rt = SlotRuntime(dec)                                              # not warmed: prepares nothing
    dec.warm(kinds=dec.WARM_HOST | dec.WARM_NO_SLOTS)
    tables = [list(range(sum(n // 256 + 1 for n in LENGTHS[:i]), sum(n // 256 + 1 for n in LENGTHS[:i + 1]))) for i in range(12)]
    for live in (range(8), range(8, 12)):                              # both launches have run once
        for i in live:
            rt.admit(i, 100 + 7 * i, LENGTHS[i], tables[i])
        rt.step()
        for i in live:
            rt.retire(i)
    kv.copy_(history)
    for i in range(12):
        rt.admit(i, 100 + 7 * i, LENGTHS[i], tables[i])
    torch.cuda.synchronize()
    hold = []
    try:
        for chunk in (1 << 30, 1 << 26, 12 << 20):
            try:
                while True:
                    hold.append(torch.empty(chunk, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                pass
        got = rt.step()
    finally:
        del hold
        torch.cuda.empty_cache()
    assert [got] == want and torch.equal(kv, kv_want)
    assert dec.status()[0] == 0
    dec.close()


@pytest.mark.parametrize("option,value,wide", [("BULK_X", 1, True), ("ROW_GEMV", 1, True), ("LMHEAD_CTAS", 0, True), ("HOST_IO", 0, True),
                                               ("SLOTS_WIDE", 0, False), ("BULK_X", 0, False), ("ROW_GEMV", 2, False),
                                               ("LMHEAD_CTAS", 64, False), ("TCGEN05", 7, False)])
def test_options_and_the_wide_steps(model, cuda_device, option, value, wide):
    """The kernels of 1 to 8 rows that an option chooses are taken at any number of slots; an option set to the value it
    has anyway chooses none."""
    from dfb_b200 import native
    g, w, history = model
    dec = H.make_decoder(w, history.clone())
    dec.set_option(getattr(native, "DFB_OPT_" + option), value)
    assert dec._lib.dfb_warm_slots(dec._handle, 2048, 0, None) == 0
    assert (_held(dec) > 0) == wide
    dec.close()


def _admitted(dec, n):
    from dfb_b200.slots import SlotRuntime
    rt, first = SlotRuntime(dec), 0
    for i in range(n):
        blocks = (LENGTHS[i] + 2) // 256 + 1           # room for three steps
        rt.admit(i, 100 + 7 * i, LENGTHS[i], list(range(first, first + blocks)))
        first += blocks
    return rt


def test_wide_step_reports_an_error_status(model, cuda_device):
    """A status that a kernel has recorded (here one of a device-pointer step whose position lies beyond the model length)
    comes back from the wide step that finds it, once; its tokens are those of a step without it."""
    from dfb_b200 import native
    g, w, history = model
    want, _ = _step(w, history, 12, None, wide=True)
    dec = H.make_decoder(w, history.clone())
    rt = _admitted(dec, 12)
    free = torch.tensor([[history.shape[2] - 1]], dtype=torch.int32, device="cuda")
    dec.enqueue_rows(torch.tensor([5], device="cuda"), torch.tensor([5000], device="cuda"), free)
    with pytest.raises(RuntimeError, match=rf"device status {native.DFB_STATUS_BAD_POSITION} .*value 5000"):
        rt.step()
    assert {i: rt.state(i)[1] for i in range(12)} == want[0] and rt.state(3)[2] == LENGTHS[3] + 1
    assert set(rt.step()) == set(range(12))
    code, st = dec.status()
    assert code == 0 and st.device_status == 0
    dec.close()


@pytest.mark.parametrize("wide", [True, False])
def test_a_row_without_a_token_is_refused(model, cuda_device, wide):
    """A sequence whose cache holds NaN has no largest logit; the step after it is refused, as the host-buffer step refuses
    a token outside the embedding table, and goes on without that sequence."""
    from dfb_b200 import native
    g, w, history = model
    kv = history.clone()
    kv[:, :, 0, 10] = float("nan")                         # a position of slot 0
    dec = H.make_decoder(w, kv)
    dec.set_option(native.DFB_OPT_SLOTS_WIDE, int(wide))
    rt = _admitted(dec, 12)
    out = rt.step()
    assert out[0] >= g.vocab and all(0 <= out[i] < g.vocab for i in range(1, 12))
    with pytest.raises(RuntimeError, match="bad argument"):
        rt.step()
    rt.retire(0)
    assert set(rt.step()) == set(range(1, 12))
    assert dec.status()[0] == 0
    dec.close()


@pytest.mark.parametrize("n", [9, 20, 32])
def test_wide_step_against_the_oracle(model, cuda_device, n):
    g, w, history = model
    got, kv_got = _step(w, history, n, None, wide=True)
    kv = history.cpu()
    first = np.cumsum([0] + [x // 256 + 1 for x in LENGTHS[:n]])
    tables = [list(range(first[i], first[i + 1])) for i in range(n)]
    logits, tokens = O.decode_step(w, kv, O.rope_cos_sin_table(g), [100 + 7 * i for i in range(n)], LENGTHS[:n], tables)
    assert float((kv_got.cpu().float() - kv.float()).abs().max()) <= 2.0 ** -5
    for i in range(n):
        assert H.token_gap_ok(logits[i].float(), got[0][i], int(tokens[i])), i


def _chunk(lengths, places=2 * 148):
    """Positions per CTA that a wide step takes: the shortest multiple of 8 from 32 on with a place for every CTA."""
    return next(c for c in range(32, 2049, 8) if sum(n // c + 1 for n in lengths) <= places)


@pytest.mark.parametrize("chunk,block_size,lengths", [
    (72, 256, [2030 - 11 * i for i in range(10)]),                # across the ends of blocks
    (112, 256, [1200 + 37 * i for i in range(20)]),
    (216, 64, [1990 - 9 * i for i in range(32)]),                 # four or five blocks each
    (232, 64, [2046 - i % 3 for i in range(32)]),                 # the longest there is
    (232, 256, [2046 - i % 3 for i in range(32)]),
    (40, 192, [511, 0, 1, 63, 64, 191, 192, 193, 2047, 1535, 1536, 1537, 1000, 999, 40, 39, 41]),
    (32, 64, [i % 8 for i in range(29)] + [2046, 1023, 2047]),    # the shortest: 64 partial results, the last of the last row among them
    (32, 64, [31, 32, 33, 7, 8, 0, 63, 64, 65])])
def test_chunks_of_every_length(cuda_device, chunk, block_size, lengths):
    """The attention of a wide step cuts the contexts into chunks that follow their sum: from 32 positions on, across block
    boundaries, several blocks long.  Two steps, between them some sequences retire and the list of chunks gets shorter, against
    launches of 8 rows: tokens, and the caches; the blocks of a row lie scattered."""
    from dfb_b200 import native
    from dfb_b200.slots import SlotRuntime
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert _chunk(lengths) == chunk
    g = H.oracle_geometry(layers=2, vocab=2048, block_size=block_size)
    w = O.make_weights(g, seed=17, norm="random").to(BF)
    signs = torch.from_numpy(np.random.Generator(np.random.Philox(key=18)).integers(0, 2, g.hidden)).to(BF) * 2 - 1
    w.embed.copy_(torch.randn(g.vocab, g.hidden, generator=torch.Generator().manual_seed(19)) * 0.5)       # (as in `model`)
    w.embed[1::2] = w.embed[0::2] * signs
    w.final_norm.copy_(signs)
    need = [min(n + 1, 2047) // block_size + 1 for n in lengths]
    order = np.random.Generator(np.random.Philox(key=8)).permutation(sum(need)).tolist()
    tables = [[order.pop() for _ in range(k)] for k in need]
    history = (torch.randn(tuple(O.new_kv_cache(g, sum(need), BF).shape), generator=torch.Generator().manual_seed(3)) * 0.5).to(BF).cuda()
    leave = [i for i in range(len(lengths)) if i % 3 == 1][:len(lengths) - 9]
    sides = []
    for wide in (1, 0):
        kv = history.clone()
        dec = H.make_decoder(w, kv)
        dec.set_option(native.DFB_OPT_SLOTS_WIDE, wide)
        rt = SlotRuntime(dec)
        for i, (n, table) in enumerate(zip(lengths, tables)):
            rt.admit(i, 100 + 7 * i, n, table)
        tokens = [rt.step()]
        for i in leave:
            rt.retire(i)
        tokens.append(rt.step())
        assert dec.status()[0] == 0
        dec.close()
        sides.append((kv, tokens))
    (kv, tokens), (want_kv, want) = sides
    assert tokens == want and set(tokens[0]) == set(range(len(lengths)))
    assert set(tokens[1]) == {i for i, n in enumerate(lengths) if i not in leave and n < 2047}
    assert torch.equal((kv != history).any(dim=-1), (want_kv != history).any(dim=-1))
    # A new value of layer 2 is a dot product of 1,024 normalised inputs, each of which may lie an ulp (2^-8) apart on the two
    # sides: 2^-8 rms, 4.5 times that among 2^16 values.  Four roundings follow (the product, two of the norm, the rotation), each
    # an ulp of the value and its rotation partner.
    new = (want_kv != history).any(dim=-1)
    got, ref = kv[new].float(), want_kv[new].float()
    pair = torch.hypot(ref[:, :64], ref[:, 64:]).repeat(1, 2)
    bound = 2.0 ** -8 * (4 * pair + 4.5 * ref.square().mean(dim=-1, keepdim=True).sqrt())
    assert bool(((got - ref).abs() <= bound).all()), float(((got - ref).abs() / bound).max())
