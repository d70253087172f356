"""Steps of 9 to 32 slots in one pass over the weights (``dfb_wide.cuh``) against the same step taken in launches of 8
rows (which a tuning option selects): one, several and all rows of the last group of 8, contexts of one token, around
chunk and block boundaries and of the full model length, sampled rows in some groups (the noise stream is the one of the
launches of 8) and an error status.  One step from the same state: the new cache rows and the tokens."""

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
        dec.set_option(native.DFB_OPT_BULK_X, 1)       # the default value; a decoder with a tuned chain steps 8 rows at a time
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
