"""The tcgen05 prefill attention kernel at its edges (64-key tiles, 128-row query tiles, both query-head ratios,
cache blocks smaller than a tile, maxima that grow along the sequence) and the line between it and the kernel for
short prompts, against the fp32 computation."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _reference(q, k, v, q_len, k_len, scale):
    """fp32 causal attention of one sequence whose last q_len of k_len positions are the queries."""
    rep = q.shape[1] // k.shape[1]
    s = torch.einsum("qhd,khd->hqk", q.float(), k.float().repeat_interleave(rep, 1)) * scale
    hidden = torch.arange(k_len)[None, :] > torch.arange(q_len)[:, None] + (k_len - q_len)
    s = s.masked_fill(hidden, float("-inf"))
    return torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), v.float().repeat_interleave(rep, 1))


@pytest.mark.parametrize("q_heads,kv_heads", [(16, 8), (8, 8), (12, 4)])
@pytest.mark.parametrize("lens,growing", [((384, 385), False), ((129, 127, 64, 65, 511, 1, 128), False), ((640, 2048), True),
                                          ((1,) * 40 + (257,), False)])
def test_fresh_prompts(cuda_device, q_heads, kv_heads, lens, growing):
    from dfb_b200.kv_store import prefill_attention

    rng = np.random.Generator(np.random.Philox(key=sum(lens) + q_heads))
    n, d = sum(lens), 128
    q, k, v = (torch.from_numpy(rng.standard_normal((n, h, d), dtype=np.float32)) for h in (q_heads, kv_heads, kv_heads))
    if growing:      # later keys score higher, so that the running maximum of a row has to be raised again and again
        k *= torch.cat([1 + torch.arange(m) / 60.0 for m in lens])[:, None, None]
    q, k, v = q.to(BF), k.to(BF), v.to(BF)
    cu = torch.tensor(np.cumsum([0, *lens]), dtype=torch.int32, device="cuda")
    got = prefill_attention(q.cuda(), k.cuda(), v.cuda(), cu, max(lens), d ** -0.5).float().cpu()
    start = 0
    for m in lens:
        want = _reference(q[start:start + m], k[start:start + m], v[start:start + m], m, m, d ** -0.5)
        assert float((got[start:start + m] - want).abs().max()) <= (2.0 ** -5 if growing else 2.0 ** -6), m
        start += m


@pytest.mark.parametrize("block_size", [4, 16, 64, 256])
@pytest.mark.parametrize("q_heads,kv_heads", [(16, 8), (8, 8)])
def test_prefix_cache_block_sizes(cuda_device, block_size, q_heads, kv_heads):
    from dfb_b200.kv_store import prefill_attention

    rng = np.random.Generator(np.random.Philox(key=block_size + q_heads))
    case, d = ((300, 44), (128, 128), (65, 1), (500, 333)), 128
    need = [-(-k // block_size) for k, _ in case]
    pool = rng.permutation(sum(need) + 2).tolist()
    kc, vc = (torch.from_numpy(rng.standard_normal((sum(need) + 2, block_size, kv_heads, d), dtype=np.float32)).to(BF)
              for _ in range(2))
    tables = [[pool.pop() for _ in range(m)] for m in need]
    q = torch.from_numpy(rng.standard_normal((sum(m for _, m in case), q_heads, d), dtype=np.float32)).to(BF)
    # what lies behind the end of a sequence in its last block never counts
    for (k_len, _), t in zip(case, tables):
        if k_len % block_size:
            vc[t[-1], k_len % block_size:] = float("nan")
    cu_q, cu_k = (torch.tensor(np.cumsum([0, *x]), dtype=torch.int32, device="cuda") for x in ([c[1] for c in case], [c[0] for c in case]))
    bt = torch.tensor([t + [0] * (max(need) - len(t)) for t in tables], dtype=torch.int32, device="cuda")
    got = prefill_attention(q.cuda(), kc.cuda(), vc.cuda(), cu_q, max(c[1] for c in case), d ** -0.5, cu_seqlens_k=cu_k,
                            block_table=bt).float().cpu()
    start = 0
    for (k_len, q_len), t in zip(case, tables):
        k, v = kc[t].flatten(0, 1)[:k_len], vc[t].flatten(0, 1)[:k_len]
        want = _reference(q[start:start + q_len], k, v, q_len, k_len, d ** -0.5)
        assert float((got[start:start + q_len] - want).abs().max()) <= 2.0 ** -6, (k_len, q_len)
        start += q_len


@pytest.mark.parametrize("q_heads,kv_heads", [(16, 8), (8, 8), (12, 4)])
@pytest.mark.parametrize("lens,growing", [((512,), False), ((385,), False), ((449,), True), ((1024,), True), ((513, 1), False),
                                          ((640, 65, 128), True), ((1088,), True)])
def test_keys_split_over_both_tiles(cuda_device, q_heads, kv_heads, lens, growing):
    """Batches small enough for the split form: odd and even numbers of key tiles, rows whose first own tile holds no
    visible key, maxima that keep growing."""
    from dfb_b200.kv_store import prefill_attention

    rng = np.random.Generator(np.random.Philox(key=sum(lens) + q_heads))
    n, d = sum(lens), 128
    q, k, v = (torch.from_numpy(rng.standard_normal((n, h, d), dtype=np.float32)) for h in (q_heads, kv_heads, kv_heads))
    if growing:
        k *= torch.cat([1 + torch.arange(m) / 60.0 for m in lens])[:, None, None]
        q -= 2.0      # scores far below zero as well as above
    q, k, v = q.to(BF), k.to(BF), v.to(BF)
    cu = torch.tensor(np.cumsum([0, *lens]), dtype=torch.int32, device="cuda")
    got = prefill_attention(q.cuda(), k.cuda(), v.cuda(), cu, max(lens), d ** -0.5).float().cpu()
    start = 0
    for m in lens:
        want = _reference(q[start:start + m], k[start:start + m], v[start:start + m], m, m, d ** -0.5)
        assert float((got[start:start + m] - want).abs().max()) <= (2.0 ** -5 if growing else 2.0 ** -6), m
        start += m


@pytest.mark.parametrize("case", [((1, 300),), ((1024, 65),), ((300, 301), (257, 64), (1, 1)), ((1600, 1100),)])
def test_keys_split_over_both_tiles_prefix_cache(cuda_device, case):
    """The same from the paged cache: (keys, queries) with odd and even numbers of key tiles and one key."""
    from dfb_b200.kv_store import prefill_attention

    case = tuple((max(a, b), min(a, b)) for a, b in case)
    rng = np.random.Generator(np.random.Philox(key=sum(k for k, _ in case)))
    d, block_size = 128, 256
    need = [-(-k // block_size) for k, _ in case]
    pool = rng.permutation(sum(need) + 2).tolist()
    kc, vc = (torch.from_numpy(rng.standard_normal((sum(need) + 2, block_size, 8, d), dtype=np.float32)).to(BF) for _ in range(2))
    tables = [[pool.pop() for _ in range(m)] for m in need]
    q = torch.from_numpy(rng.standard_normal((sum(m for _, m in case), 16, d), dtype=np.float32)).to(BF)
    for (k_len, _), t in zip(case, tables):
        if k_len % block_size:
            vc[t[-1], k_len % block_size:] = float("nan")      # what lies behind the end never counts
    cu_q, cu_k = (torch.tensor(np.cumsum([0, *x]), dtype=torch.int32, device="cuda") for x in ([c[1] for c in case], [c[0] for c in case]))
    bt = torch.tensor([t + [0] * (max(need) - len(t)) for t in tables], dtype=torch.int32, device="cuda")
    got = prefill_attention(q.cuda(), kc.cuda(), vc.cuda(), cu_q, max(m for _, m in case), d ** -0.5, cu_seqlens_k=cu_k,
                            block_table=bt).float().cpu()
    start = 0
    for (k_len, m), t in zip(case, tables):
        flat = [x[t].reshape(-1, 8, d)[:k_len] for x in (kc, vc)]
        want = _reference(q[start:start + m], *flat, m, k_len, d ** -0.5)
        assert float((got[start:start + m] - want).abs().max()) <= 2.0 ** -6
        start += m


@pytest.mark.parametrize("q_heads,kv_heads,new,cached", [
    (16, 8, (512,), (0,)), (16, 8, (700,), (1024,)),                    # keys split over both tiles: fresh, paged
    (16, 8, (512,) * 4, (0,) * 4), (24, 24, (300,) * 5, (0,) * 5),       # head pairs, single heads
    (16, 8, (300,) * 12, (256,) * 12), (24, 24, (300,) * 5, (256,) * 5)])
def test_error_against_64_bits(cuda_device, q_heads, kv_heads, new, cached):
    """The roundings of the result are those of the computation as it is defined: probabilities rounded to bf16 relative to
    the row's maximum (which is 1 exactly), their sum over the rounded values, the result rounded once.  Scores of 4 times
    the usual spread, so that few keys carry a row.  The 2-norm of the error may exceed that of the same roundings
    emulated in 64 bits by 2 % (it repeats to 0.5 % from seed to seed); an unrounded sum costs 11 % to 24 %, a maximum
    that lags behind 2 % to 8 %."""
    from dfb_b200.kv_store import prefill_attention

    gen = torch.Generator(device="cuda").manual_seed(sum(new) + q_heads)
    d, bs, total = 128, 256, [a + b for a, b in zip(new, cached)]
    q = torch.empty(sum(new), q_heads, d, device="cuda").normal_(generator=gen).to(BF)
    ks = [(4 * torch.empty(n, kv_heads, d, device="cuda").normal_(generator=gen)).to(BF) for n in total]
    vs = [torch.empty(n, kv_heads, d, device="cuda").normal_(generator=gen).to(BF) for n in total]
    cu_q, cu_k = (torch.tensor(np.cumsum([0, *x]), dtype=torch.int32, device="cuda") for x in (new, total))
    if any(cached):
        need = [-(-n // bs) for n in total]
        kc, vc = (torch.zeros(sum(need), bs, kv_heads, d, dtype=BF, device="cuda") for _ in range(2))
        first = np.cumsum([0, *need])
        for i, n in enumerate(total):
            kc.flatten(0, 1)[first[i] * bs:first[i] * bs + n] = ks[i]
            vc.flatten(0, 1)[first[i] * bs:first[i] * bs + n] = vs[i]
        bt = torch.tensor([[first[i] + c if c < m else 0 for c in range(max(need))] for i, m in enumerate(need)],
                          dtype=torch.int32, device="cuda")
        got = prefill_attention(q, kc, vc, cu_q, max(new), d ** -0.5, cu_seqlens_k=cu_k, block_table=bt)
    else:
        got = prefill_attention(q, torch.cat(ks), torch.cat(vs), cu_q, max(new), d ** -0.5)
    err, emulated = 0.0, 0.0
    for i, n in enumerate(new):
        rows = slice(sum(new[:i]), sum(new[:i]) + n)
        hidden = torch.arange(total[i], device="cuda")[None] > torch.arange(n, device="cuda")[:, None] + cached[i]
        for h in range(q_heads):
            kh, vh = (x[i][:, h * kv_heads // q_heads].double() for x in (ks, vs))
            s = (q[rows, h].double() @ kh.T * d ** -0.5).masked_fill(hidden, float("-inf"))
            p = torch.exp(s - s.max(-1, keepdim=True).values)
            exact = p @ vh / p.sum(-1, keepdim=True)
            r = p.to(BF).double()
            emulated += float(((r @ vh / r.sum(-1, keepdim=True)).to(BF).double() - exact).square().sum())
            err += float((got[rows, h].double() - exact).square().sum())
    assert err ** 0.5 <= 1.02 * emulated ** 0.5, (err / emulated) ** 0.5


@pytest.mark.parametrize("scale", [-0.09, 0.0])
@pytest.mark.parametrize("new,cached", [((100,), (0,)), ((300, 513), (0, 0)), ((640,) * 4, (0,) * 4),       # short, split, pairs
                                        ((300, 65), (512, 256)), ((300,) * 12, (256,) * 12)])
def test_scale_of_either_sign(cuda_device, scale, new, cached):
    """A scale that is not positive: the largest score is the smallest product, or all scores are equal."""
    from dfb_b200.kv_store import prefill_attention

    rng = np.random.Generator(np.random.Philox(key=sum(new)))
    d, bs, total = 128, 256, [a + b for a, b in zip(new, cached)]
    q = torch.from_numpy(rng.standard_normal((sum(new), 16, d), dtype=np.float32)).to(BF)
    ks, vs = ([torch.from_numpy(rng.standard_normal((n, 8, d), dtype=np.float32)).to(BF) for n in total] for _ in range(2))
    cu_q, cu_k = (torch.tensor(np.cumsum([0, *x]), dtype=torch.int32, device="cuda") for x in (new, total))
    if any(cached):
        need = [-(-n // bs) for n in total]
        kc, vc = (torch.zeros(sum(need), bs, 8, d, dtype=BF) for _ in range(2))
        first = np.cumsum([0, *need])
        for i, n in enumerate(total):
            kc.flatten(0, 1)[first[i] * bs:first[i] * bs + n] = ks[i]
            vc.flatten(0, 1)[first[i] * bs:first[i] * bs + n] = vs[i]
        bt = torch.tensor([[first[i] + c if c < m else 0 for c in range(max(need))] for i, m in enumerate(need)],
                          dtype=torch.int32, device="cuda")
        got = prefill_attention(q.cuda(), kc.cuda(), vc.cuda(), cu_q, max(new), scale, cu_seqlens_k=cu_k, block_table=bt)
    else:
        got = prefill_attention(q.cuda(), torch.cat(ks).cuda(), torch.cat(vs).cuda(), cu_q, max(new), scale)
    start = 0
    for i, n in enumerate(new):
        want = _reference(q[start:start + n], ks[i], vs[i], n, total[i], scale)
        assert float((got[start:start + n].float().cpu() - want).abs().max()) <= 2.0 ** -6
        start += n


def _split(lens, q_heads, longest, rows_known=True):
    """The launcher's rule: whether the keys of an item go to both tiles."""
    tiles = len(lens) * -(-longest // 128)
    if rows_known:
        tiles = min(tiles, sum(lens) // 128 + len(lens))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return tiles * q_heads <= (2 if longest >= 1024 else 1) * sms


@pytest.mark.parametrize("block_size", [4, 16, 64, 256])
@pytest.mark.parametrize("q_heads,kv_heads", [(16, 8), (24, 24)])
@pytest.mark.parametrize("bad", [False, True])
def test_prefix_cache_above_the_line(cuda_device, block_size, q_heads, kv_heads, bad):
    """Batches of the prefix cache that are too large for the split form: head pairs and single heads, blocks smaller than
    a key tile, NaN behind the ends, a block id outside the cache (its keys are read as zeros, and reported)."""
    from dfb_b200 import native
    from dfb_b200.kv_store import prefill_attention

    rng = np.random.Generator(np.random.Philox(key=block_size + q_heads))
    case = [(129 + 16 * i + extra, 129 + 14 * i) for i, extra in enumerate((0, 1, 300, 64, 128, 7, 512, 63, 256, 65, 40, 1000))]
    d, lens = 128, [q for _, q in case]
    assert not _split(lens, q_heads, max(lens))
    need = [-(-k // block_size) for k, _ in case]
    pool = rng.permutation(sum(need) + 2).tolist()
    kc, vc = (torch.from_numpy(rng.standard_normal((sum(need) + 2, block_size, kv_heads, d), dtype=np.float32)).to(BF)
              for _ in range(2))
    tables = [[pool.pop() for _ in range(m)] for m in need]
    q = torch.from_numpy(rng.standard_normal((sum(lens), q_heads, d), dtype=np.float32)).to(BF)
    for (k_len, _), t in zip(case, tables):
        if k_len % block_size:
            vc[t[-1], k_len % block_size:] = float("nan")
    cu_q, cu_k = (torch.tensor(np.cumsum([0, *x]), dtype=torch.int32, device="cuda") for x in (lens, [k for k, _ in case]))
    bt = torch.tensor([t + [0] * (max(need) - len(t)) for t in tables], dtype=torch.int32)
    where = (5, 100 // block_size)
    if bad:
        bt[where] = sum(need) + 2
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    got = prefill_attention(q.cuda(), kc.cuda(), vc.cuda(), cu_q, max(lens), d ** -0.5, cu_seqlens_k=cu_k,
                            block_table=bt.cuda(), status=status).float().cpu()
    start = 0
    for i, ((k_len, q_len), t) in enumerate(zip(case, tables)):
        k, v = (x[t].flatten(0, 1)[:k_len].clone() for x in (kc, vc))
        if bad and i == where[0]:
            for x in (k, v):
                x[where[1] * block_size:(where[1] + 1) * block_size] = 0
        want = _reference(q[start:start + q_len], k, v, q_len, k_len, d ** -0.5)
        assert float((got[start:start + q_len] - want).abs().max()) <= 2.0 ** -6, (k_len, q_len)
        start += q_len
    assert status.tolist()[:1] + status.tolist()[2:] == ([native.DFB_STATUS_BAD_BLOCK, where[0], sum(need) + 2] if bad else [0, 0, 0])


@pytest.mark.parametrize("known", [True, False])
@pytest.mark.parametrize("q_heads,kv_heads,lens", [
    (16, 8, (264, 65, 129, 200)), (16, 8, (449,)), (8, 8, (511, 8, 136)),                     # split form
    (16, 8, (520, 193, 640, 64, 321, 72)), (24, 24, (136, 300, 257, 255, 129)), (16, 8, (2048, 1, 1025, 512, 319, 200))])
def test_entry_points_with_and_without_sizes(cuda_device, known, q_heads, kv_heads, lens):
    """``dfb_prefill_attention`` does not know where the tensors end and fetches the ends of the sequences in boxes of 8 rows
    and pieces; ``dfb_prefill_attention_rows`` may be told.  Ends around multiples of 8 and 64, the last one at the
    tensors' end, NaN in the rows of the second sequence (or behind the only one's)."""
    from dfb_b200 import native

    lib, d, n = native.lib(), 128, sum(lens)
    gen = torch.Generator().manual_seed(n + q_heads)
    pad = 0 if len(lens) > 1 else 64             # rows of nobody behind a single sequence
    q, k, v = (torch.randn(n + pad, h, d, generator=gen).to(BF) for h in (q_heads, kv_heads, kv_heads))
    spoilt = range(lens[0], lens[0] + (lens[1] if pad == 0 else pad))
    for x in (k, v):
        x[spoilt.start:spoilt.stop] = float("nan")
    dev = [x.cuda() for x in (q, k, v)]
    out = torch.zeros(n + pad, q_heads, d, dtype=BF, device="cuda")
    cu = torch.tensor(np.cumsum([0, *lens]), dtype=torch.int32, device="cuda")
    args = [*(x.data_ptr() for x in dev), out.data_ptr(), cu.data_ptr(), None, len(lens), max(lens), q_heads * d, kv_heads * d,
            kv_heads * d, q_heads * d, q_heads, kv_heads, d, d ** -0.5, None, 0, 0, 0, None]
    stream = torch.cuda.current_stream().cuda_stream
    code = lib.dfb_prefill_attention_rows(*args, n + pad, n + pad, stream) if known else lib.dfb_prefill_attention(*args, stream)
    assert code == 0
    got, start = out.float().cpu(), 0
    for i, m in enumerate(lens):
        rows = slice(start, start + m)
        if i != 1:
            want = _reference(q[rows], k[rows], v[rows], m, m, d ** -0.5)
            assert float((got[rows] - want).abs().max()) <= 2.0 ** -6, (i, m)
        start += m
    assert float(got[n:].abs().sum()) == 0.0
