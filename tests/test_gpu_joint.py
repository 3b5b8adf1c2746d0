"""The joint log-likelihood against the oracle at the kernel's limits: words of
0 to several thousand tokens (a warp's, a whole CTA's from 2048 tokens, and
words split over work items), counts beyond the tabulated ones, K at both ends.
Both sides sum FP64 terms: 1e-10 relative, as in the other joint tests."""
from __future__ import annotations

import numpy as np
import pytest

import culda_cgs_b200 as cb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,item_tokens", [(32, 0), (32, 300), (1024, 0), (1024, 2500), (4096, 0)])
def test_joint_matches_oracle(k, item_tokens):
    rng = np.random.default_rng(k + item_tokens)
    lens = np.concatenate([[0, 1, 2047, 2048, 2049, 6000, 0], rng.integers(0, 60, 400), [33, 0]])
    docs = 300
    word = np.repeat(np.arange(len(lens)), lens)
    doc = rng.integers(0, docs, len(word)) * rng.integers(0, 2, len(word))  # half the tokens in doc 0
    order = np.lexsort((doc, word))
    ids = doc[order].astype(np.int32)
    doc_ptr = np.concatenate([[0], np.cumsum(np.bincount(doc, minlength=docs))])
    word_ptr = np.concatenate([[0], np.cumsum(lens)])
    c = cb.Corpus.from_arrays(doc_ptr, word_ptr, ids)
    # topic 3 holds most tokens, so some counts are far past the table
    z = np.where(rng.random(len(word)) < 0.7, 3, rng.integers(0, k, len(word))).astype(np.uint16)
    with cb.LDA(c, k, 0.05, 0.01, item_tokens=item_tokens) as m:
        m.set_topics(z)
        want = O.Snapshot.build(c.word_ptr, c.doc_ids, c.doc_ptr, z, k, m.alpha, m.beta).loglik_joint()
        got = m.loglik_joint()
        assert got == pytest.approx(want, rel=1e-10)
        assert m.loglik_joint() == got  # fixed assignment: the same bits again
