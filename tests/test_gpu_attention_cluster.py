"""The cluster attention kernel (``dfb_attncluster.cuh``) at the edges of its pieces and passes: the grids for which the
decoder picks clusters of 2, 4 and 8 CTAs, contexts around multiples of 16 positions per CTA, of 128 positions per
pass and of a cache block, rows that leave most CTAs of their cluster without a position, against the fp32 oracle."""

import numpy as np
import pytest
import torch

from tests.test_gpu_kernels import _attention_case, small  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctx_lens", [
    (129, 1, 256, 31, 33), (255, 192, 2, 160, 161, 130, 32, 16),                                  # clusters of 2
    (257, 64, 512), (511, 1, 65, 513 - 64, 320), (512, 257, 17, 63, 449, 384, 400, 511),          # of 4, one pass
    (1281, 5, 2048, 1024), (2047, 127, 129, 1290),                                                # of 8
    (2048, 1, 513, 1025, 256, 700, 1536, 2033), (1024, 15, 640, 1000, 897, 3)])                   # of 4, several passes
@pytest.mark.parametrize("scattered", [False, True])
def test_cluster_attention(small, ctx_lens, scattered):  # noqa: F811
    g, w = small
    perm = np.random.Generator(np.random.Philox(key=19)).permutation(64).tolist() if scattered else None
    active = [i % 3 != 1 for i in range(len(ctx_lens))] if scattered else None
    out, want, kv_got, kv_want, _ = _attention_case(g, w, len(ctx_lens), list(ctx_lens), seed=81, perm=perm,
                                                    row_active=[int(x) for x in active] if active else None)
    assert float((out.float() - want.float()).abs().max()) <= 2.0 ** -6
    assert torch.equal(kv_got, kv_want)            # the active rows' new K/V bit-exactly, nothing else touched


def test_attention_options_from_the_environment(cuda_device, monkeypatch):
    """The environment's initial value of an attention option counts like one that is set: the kernel it speaks of (the
    streaming one, whose order of sums shows in the caches' last bits) runs where the cluster kernel would."""
    from dfb_b200 import native
    from oracle import qwen3_decode as O
    from tests import harness as H

    g = H.oracle_geometry(layers=3, vocab=2048)
    w = O.make_weights(g, seed=23, norm="random").to(torch.bfloat16)
    history = torch.randn(tuple(O.new_kv_cache(g, 16, torch.bfloat16).shape), generator=torch.Generator().manual_seed(24))
    contexts = [130, 399, 200, 256, 257, 300, 171, 380]

    def caches(env, opt):
        if env:
            monkeypatch.setenv("DFB_ATTN_RING32", "1")
        kv = history.to(torch.bfloat16).cuda()
        dec = H.make_decoder(w, kv)
        if opt:
            dec.set_option(native.DFB_OPT_ATTN_RING32, 1)
        dec.decode_host([7 * r for r in range(8)], contexts, [[2 * r, 2 * r + 1] for r in range(8)])
        dec.close()
        monkeypatch.delenv("DFB_ATTN_RING32", raising=False)
        return kv

    default, chosen = caches(False, False), caches(False, True)
    assert not torch.equal(default, chosen)                 # another kernel, another order of sums
    assert torch.equal(caches(True, False), chosen)
