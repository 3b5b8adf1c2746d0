"""Work items of at most 32 tokens are sampled by a kernel of their own (a warp
per item) when they come last in the work list, and short lists by CTAs of 16
warps instead of 4.  The draws must equal, bit for bit, those of the narrow CTAs
that the kernel-level entry point uses for every item of a long list in another
order: the same corpus in the same token order, topics, uniforms and items."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import culda_cgs_b200 as cb
from culda_cgs_b200 import _ffi
from oracle import oracle as O

from kernel_api import doc_term, host, prepare, ptr, sample_args, update_theta

pytestmark = pytest.mark.gpu


def corpus(rng, lens, docs, long_docs):
    """Words of the given token counts over `docs` documents, a share of the
    tokens in the `long_docs` longest, so rows run from one block of 32 entries
    to more than the walk's budget for 32 segments."""
    word = np.repeat(np.arange(len(lens)), lens)
    doc = np.where(rng.random(len(word)) < 0.5, rng.integers(0, max(1, long_docs), len(word)),
                   rng.integers(0, docs, len(word)))
    order = np.lexsort((doc, word))
    return cb.Corpus.from_arrays(np.concatenate([[0], np.cumsum(np.bincount(doc, minlength=docs))]),
                                 np.concatenate([[0], np.cumsum(lens)]), doc[order].astype(np.int32))


@pytest.mark.parametrize("k", [32, 64, 512, 1024, 2048, 4096])
@pytest.mark.parametrize("long_docs,large", [(1, 0), (12, 150), (12, 700)])
@pytest.mark.parametrize("shuffled", [False, True])
def test_small_items_draw_as_the_cta_kernel(k, long_docs, large, shuffled):
    import torch

    rng = np.random.default_rng(k + long_docs)
    lens = np.concatenate([np.arange(0, 70), rng.integers(1, 33, 3000), [1500], np.full(300, 1), [33, 32, 31],
                           rng.integers(33, 90, large)])
    c = corpus(rng, lens, 400, long_docs)
    z = O.init_topics(c.num_tokens, k, 5)
    with cb.LDA(c, k, 0.05, 0.01, seed=9, flags=cb.CULDA_FLAG_NO_REORDER) as m:
        m.set_topics(z)
        got, ll = m.sample_snapshot(4)
        item_tokens = m.info()["item_tokens"]
    p = prepare(c, k, 0.05, 0.01, z, item_tokens=item_tokens)
    assert update_theta(p) == 0
    if shuffled:  # a small item first: every item takes a CTA
        items = np.frombuffer(bytes(p.items), dtype=np.uint8).reshape(p.num_items, -1)
        p.d["items"] = torch.from_numpy(np.ascontiguousarray(items[::-1])).cuda()
    a = sample_args(p, seed=9, iteration=4, group_lanes=_ffi.CULDA_SAMPLER_FLAT)
    ws = torch.zeros(cb.lib().culda_sample_workspace(k, p.num_items, p.num_hot) // 4 + 64, dtype=torch.int32,
                     device="cuda")
    assert cb.lib().culda_sample(C.byref(a), ptr(ws), ws.numel() * 4, None) == 0
    torch.cuda.synchronize()
    assert int(p.d["err"].item()) == 0
    assert np.array_equal(got, host(p.d["z_out"], np.uint16))
    want = C.c_double()
    assert cb.lib().culda_loglik(ptr(p.d["ll"]), doc_term(p), c.num_tokens, C.byref(want), None) == 0
    assert ll == pytest.approx(want.value, rel=1e-12)  # FP64 sums in another order
