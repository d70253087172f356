"""The work that a user of this framework has it do, as timed cases.

Everything goes through the public entry points, the way an engine's model
runner calls them: ``MegakernelBackend.decode`` / ``decode_batch`` for decode
steps, ``StreamDecoder.decode_burst`` for several steps per call,
``SlotRuntime`` for a set of sequences that is wider than one launch, and
``kv_store.prefill_attention`` / ``store_kvcache`` for the prefill side of the
shared paged cache.  The model is the one the backend admits (28 layers, hidden
1024, 16 query / 8 KV heads, vocabulary 151,936, blocks of 256 tokens, up to
2,048 tokens per sequence, up to 8 rows per call, 32 slots).

    listed()              the named cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   what the caller has in hand before the call
    run(state)            one call, and what it computes
    work(case)            bytes and operations the call cannot do without
    tolerance(case)       how far another correct implementation may be off
"""

from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import torch

import __graft_entry__

__graft_entry__.load_package()

from dfb_b200 import QWEN3_06B, MegakernelBackend  # noqa: E402
from dfb_b200.kv_store import prefill_attention, store_kvcache  # noqa: E402
from dfb_b200.slots import SlotRuntime  # noqa: E402
from dfb_b200.synthetic import nano_model_view  # noqa: E402
from dfb_b200.weights import DecoderWeights, LayerTensors, rope_cos_sin_table  # noqa: E402

G = QWEN3_06B
BF = torch.bfloat16
MAX_PROMPT = 2048          # tokens of one sequence (max_model_len)
MAX_PROMPT_TOKENS = 16384  # prompt tokens of one prefill batch


def listed():
    return [
        # a short prompt's K / V rows into the cache: one call per layer of a prefill, dominated by the call itself
        {"name": "store-37", "kind": "store", "tokens": 37},
        # the same for a full prefill batch
        {"name": "store-16384", "kind": "store", "tokens": 16384},
        # attention of one ordinary prompt (the length of the benchmark configurations)
        {"name": "prompt-512", "kind": "prompt", "prompts": "512", "cached": ""},
        # a full prefill batch of uneven prompts, some of them at the model length
        {"name": "prompts-ragged", "kind": "prompt", "prompts": "2048,1531,37,2047,977,1,2048,300,1290,2000,701,1800,64",
         "cached": ""},
        # prompts whose first blocks were found in the prefix cache: keys come from the paged cache
        {"name": "prompts-cached", "kind": "prompt", "prompts": "129,700,64,31,1000", "cached": "512,1024,1792,256,768"},
        # one user chatting, at the start of a conversation: latency of one token
        {"name": "decode-1-short", "kind": "decode", "contexts": "33", "sampled": False},
        # and far into it
        {"name": "decode-1-long", "kind": "decode", "contexts": "1405", "sampled": False},
        # a few users, sampling with temperatures
        {"name": "decode-3-sampled", "kind": "decode", "contexts": "418,97,650", "sampled": True},
        # a full call in the middle of 512-token prompts' answers (the batch sweep's largest point)
        {"name": "decode-8", "kind": "decode", "contexts": "513,576,530,639,601,555,520,617", "sampled": False},
        # a full call of long, uneven contexts: the KV cache outweighs the weights
        {"name": "decode-8-long", "kind": "decode", "contexts": "1840,735,1773,2040,1290,960,1511,256", "sampled": False},
        # offline generation: many steps per call, tokens fed back on the device
        {"name": "burst-2x64", "kind": "burst", "contexts": "300,905", "steps": 64},
        # continuous batching over more sequences than one launch takes: admission, then eight steps
        {"name": "slots-20", "kind": "slots",
         "contexts": "40,700,255,1300,64,512,901,17,330,128,1020,77,450,600,5,210,860,1500,390,95", "steps": 8},
    ]


def _log_int(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _some(rng, n, lo, hi):
    return ",".join(str(_log_int(rng, lo, hi)) for _ in range(n))


def draw(rng):
    kind = rng.choice(["store", "prompt", "prompt", "cached", "decode", "decode", "decode", "burst", "slots"])
    if kind == "store":
        return {"kind": kind, "tokens": _log_int(rng, 1, MAX_PROMPT_TOKENS)}
    if kind == "prompt":
        lens, left = [], MAX_PROMPT_TOKENS - 1548
        for _ in range(_log_int(rng, 1, 12)):
            n = min(_log_int(rng, 3, MAX_PROMPT), left)
            if n > 0:
                lens.append(n)
                left -= n
        return {"kind": kind, "prompts": ",".join(map(str, lens)), "cached": ""}
    if kind == "cached":
        new, old = [], []
        for _ in range(rng.randint(1, 6)):
            blocks = rng.randint(1, 7)                     # whole blocks of the prefix cache
            old.append(blocks * G.block_size)
            new.append(_log_int(rng, 1, MAX_PROMPT - blocks * G.block_size))
        return {"kind": "prompt", "prompts": ",".join(map(str, new)), "cached": ",".join(map(str, old))}
    if kind == "decode":
        rows = rng.choice([1, 1, 2, 3, 4, 5, 6, 7, 8])
        return {"kind": kind, "contexts": _some(rng, rows, 2, G.max_model_len), "sampled": rng.random() < 0.25}
    if kind == "burst":
        steps = _log_int(rng, 4, 32)
        return {"kind": kind, "contexts": _some(rng, rng.randint(1, 4), 2, G.max_model_len - steps), "steps": steps}
    return {"kind": kind, "contexts": _some(rng, rng.randint(2, 32), 2, G.max_model_len - 8), "steps": rng.randint(3, 8)}


def _ints(text):
    return [int(x) for x in text.split(",") if x]


# ---- inputs ------------------------------------------------------------------------------------------------
def _weights(gen):
    """Random weights under which the model behaves as a trained one does: the matrices that write to the residual
    stream are scaled by 1 / sqrt(2 layers), so that rounding differences stay small over the depth, and the
    next token has a clear margin: the embedding rows of an even and the following odd token are one another's
    images under the final norm's signs, so each predicts the other."""
    def mat(rows, cols, std=0.02):
        return torch.empty(rows, cols, dtype=BF, device="cuda").normal_(0.0, std, generator=gen)

    def vec(n):
        return torch.empty(n, dtype=torch.float32, device="cuda").normal_(1.0, 0.1, generator=gen).to(BF)

    out_std = 0.02 / math.sqrt(2 * G.layers)
    signs = torch.randint(0, 2, (G.hidden,), device="cuda", generator=gen).to(BF) * 2 - 1
    embed = mat(G.vocab, G.hidden, 0.125)
    embed[1::2] = embed[0::2] * signs
    layers = [LayerTensors(ln_in=vec(G.hidden), wqkv=mat(G.qkv_rows, G.hidden), q_norm=vec(G.head_dim),
                           k_norm=vec(G.head_dim), wo=mat(G.hidden, G.q_size, out_std), ln_post=vec(G.hidden),
                           wgu=mat(2 * G.intermediate, G.hidden), wd=mat(G.hidden, G.intermediate, out_std))
              for _ in range(G.layers)]
    return DecoderWeights(G, embed, layers, signs, rope_cos_sin_table(G).cuda())


def _backend(gen, contexts, steps, sampled=False):
    """A backend over the model and a paged cache that already holds the contexts' keys (unit RMS, as after their
    norm) and values, with the blocks of the sequences scattered over the pool."""
    need = [-(-(n + steps) // G.block_size) for n in contexts]
    blocks = sum(need) + 8
    kv = torch.empty(2, G.layers, blocks, G.block_size, G.kv_heads, G.head_dim, dtype=BF, device="cuda")
    kv[0].normal_(0.0, 1.0, generator=gen)
    kv[1].normal_(0.0, 0.64, generator=gen)
    order = torch.randperm(blocks, device="cuda", generator=gen).tolist()
    tables = [[order.pop() for _ in range(n)] for n in need]
    weights = _weights(gen)
    model, hf = nano_model_view(weights)
    config = SimpleNamespace(hf_config=hf, max_model_len=G.max_model_len, max_num_seqs=8, tensor_parallel_size=1,
                             kvcache_block_size=G.block_size, megakernel_sampling="batch" if sampled else False)
    backend = MegakernelBackend(config, model)
    backend.set_kv_cache(kv)
    backend.ensure_ready()
    ids = torch.randint(0, G.vocab, (len(contexts),), device="cuda", generator=gen).tolist()
    return SimpleNamespace(backend=backend, kv=kv, tables=tables, ids=ids, weights=weights)


class _Sequence:
    """What the backend reads of a scheduler's sequence."""

    def __init__(self, length, last_token):
        self.length, self.last_token, self.is_greedy, self.temperature = length, last_token, True, 0.0

    def __len__(self):
        return self.length


def _prepare_decode(case, gen):
    contexts = _ints(case["contexts"])       # tokens a row attends to in this step, its new token included
    s = _backend(gen, contexts, 0, case["sampled"])
    if len(contexts) == 1 and not case["sampled"]:
        s.kind, s.seq = "decode", _Sequence(contexts[0], s.ids[0])
        return s
    s.kind = "decode_batch"
    s.input_ids = torch.tensor(s.ids, dtype=torch.int64, device="cuda")
    s.positions = torch.tensor([n - 1 for n in contexts], dtype=torch.int64, device="cuda")
    width = max(len(t) for t in s.tables)
    s.block_tables = torch.tensor([t + [0] * (width - len(t)) for t in s.tables], dtype=torch.int32, device="cuda")
    s.temperatures = None
    if case["sampled"]:
        s.temperatures = torch.empty(len(contexts), device="cuda").uniform_(0.6, 1.0, generator=gen)
    return s


def _prepare_prompt(case, gen):
    new, old = _ints(case["prompts"]), _ints(case["cached"])
    n, d, h = sum(new), G.head_dim, G.kv_heads
    s = SimpleNamespace(kind="prompt", cu_k=None, table=None, longest=max(new))
    # queries and keys as their norms leave them (contiguous); values as a view of the fused projection's output
    s.q = torch.empty(n, G.q_heads, d, dtype=BF, device="cuda").normal_(0.0, 1.0, generator=gen)
    qkv = torch.empty(n, G.qkv_rows, dtype=BF, device="cuda").normal_(0.0, 0.64, generator=gen)
    s.k = torch.empty(n, h, d, dtype=BF, device="cuda").normal_(0.0, 1.0, generator=gen)
    s.v = qkv[:, G.q_size + G.kv_size:].view(n, h, d)
    s.cu_q = torch.tensor(np.cumsum([0] + new), dtype=torch.int32, device="cuda")
    if old:
        total = [a + b for a, b in zip(new, old)]
        need = [-(-t // G.block_size) for t in total]
        blocks = sum(need) + 8
        s.k = torch.empty(blocks, G.block_size, h, d, dtype=BF, device="cuda").normal_(0.0, 1.0, generator=gen)
        s.v = torch.empty(blocks, G.block_size, h, d, dtype=BF, device="cuda").normal_(0.0, 0.64, generator=gen)
        order = torch.randperm(blocks, device="cuda", generator=gen).tolist()
        tables = [[order.pop() for _ in range(k)] for k in need]
        s.table = torch.tensor([t + [0] * (max(need) - len(t)) for t in tables], dtype=torch.int32, device="cuda")
        s.cu_k = torch.tensor(np.cumsum([0] + total), dtype=torch.int32, device="cuda")
    return s


def _prepare_store(case, gen):
    n, h, d = case["tokens"], G.kv_heads, G.head_dim
    qkv = torch.empty(n, G.qkv_rows, dtype=BF, device="cuda").normal_(0.0, 0.64, generator=gen)
    blocks = -(-n // G.block_size) + 8
    order = torch.randperm(blocks, device="cuda", generator=gen)
    tokens = torch.arange(n, device="cuda")
    return SimpleNamespace(
        kind="store", key=torch.empty(n, h, d, dtype=BF, device="cuda").normal_(0.0, 1.0, generator=gen),
        value=qkv[:, G.q_size + G.kv_size:].view(n, h, d),
        k_cache=torch.zeros(blocks, G.block_size, h, d, dtype=BF, device="cuda"),
        v_cache=torch.zeros(blocks, G.block_size, h, d, dtype=BF, device="cuda"),
        slots=(order[tokens // G.block_size] * G.block_size + tokens % G.block_size).to(torch.int32))


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kind = case["kind"]
    if kind == "store":
        return _prepare_store(case, gen)
    if kind == "prompt":
        return _prepare_prompt(case, gen)
    if kind == "decode":
        return _prepare_decode(case, gen)
    s = _backend(gen, _ints(case["contexts"]), case["steps"])
    s.kind, s.steps, s.positions = kind, case["steps"], [n - 1 for n in _ints(case["contexts"])]
    if kind == "slots":
        s.runtime = SlotRuntime(s.backend.decoder)
    return s


# ---- one call ----------------------------------------------------------------------------------------------
def _run_slots(s):
    """A short serve: every sequence is admitted to its slot, then the live slots step together.  The tokens come
    back as the callback sees them; a slot is admitted again by the next call, at the same position."""
    for i, table in enumerate(s.tables):
        s.runtime.admit(i, s.ids[i], s.positions[i], table)
    steps = []

    def on_tokens(tokens):
        steps.append([tokens[i] for i in range(len(s.tables))])
        return False

    s.runtime.run(s.steps, on_tokens)
    return np.array(steps)


def run(s):
    if s.kind == "store":
        store_kvcache(s.key, s.value, s.k_cache, s.v_cache, s.slots)
        return {"k_cache": s.k_cache, "v_cache": s.v_cache}
    if s.kind == "prompt":
        return prefill_attention(s.q, s.k, s.v, s.cu_q, s.longest, G.head_dim ** -0.5, cu_seqlens_k=s.cu_k,
                                 block_table=s.table)
    if s.kind == "decode":
        tokens = s.backend.decode(s.seq, s.tables[0])
    elif s.kind == "decode_batch":
        tokens = s.backend.decode_batch(s.input_ids, s.positions, s.block_tables, temperatures=s.temperatures)
    elif s.kind == "burst":
        tokens = np.array(s.backend.decoder.decode_burst(s.ids, s.positions, s.tables, s.steps))
    else:
        tokens = _run_slots(s)
    return {"tokens": tokens, "k_cache": s.kv[0], "v_cache": s.kv[1]}


# ---- what a call cannot do without ---------------------------------------------------------------------------
def work(case):
    kind, d = case["kind"], G.head_dim
    if kind == "store":     # K and V rows read once and written once, one slot index each
        return {"bytes": case["tokens"] * (4 * 2 * G.kv_size + 4), "flops": 0}
    if kind == "prompt":
        new, old = _ints(case["prompts"]), _ints(case["cached"])
        old = old or [0] * len(new)
        pairs = sum(n * o + n * (n + 1) // 2 for n, o in zip(new, old))
        nbytes = 2 * (2 * sum(new) * G.q_size + 2 * (sum(new) + sum(old)) * G.kv_size)
        return {"bytes": nbytes, "flops": 4 * pairs * d * G.q_heads}
    contexts, steps = _ints(case["contexts"]), case.get("steps", 1)
    rows = len(contexts)
    attended = steps * sum(contexts) + rows * steps * (steps - 1) // 2
    nbytes = steps * G.weight_bytes_per_step() + (attended + rows * steps) * G.kv_bytes_per_token()
    flops = rows * steps * G.weight_bytes_per_step() + 4 * attended * d * G.q_heads * G.layers
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Moving rows is exact.  Attention returns bf16 (2**-9 relative rounding of its result and of the
    probabilities).  A decode step returns whole token ids, which have to be the same, and the caches, whose new
    rows went through 28 layers of bf16 activations (1 % of a new row, single values up to an eighth)."""
    if case["kind"] == "store":
        return "exact"
    if case["kind"] == "prompt":
        return {"rel": 1e-2, "max": 5e-2}
    return {"rel": 1e-2, "max": 2.5e-1, "differ": 0.0}
