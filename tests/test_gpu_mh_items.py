"""A Metropolis-Hastings pass draws the same topics however the words are cut
into work items: by a CTA (256 tokens or more), by a warp, split over items (the
hot rows), with the proposal's block table within one 128-byte line (K <= 1024)
or past it, and with an odd number of steps.  Draws are exact."""
from __future__ import annotations

import numpy as np
import pytest

import culda_cgs_b200 as cb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [128, 1024, 1152])
@pytest.mark.parametrize("proposal", [False, True])
def test_pass_does_not_depend_on_the_items(k, proposal):
    rng = np.random.default_rng(k)
    lens = np.concatenate([[0, 1, 255, 256, 257, 2000], rng.integers(0, 70, 400)])
    docs = 150
    word = np.repeat(np.arange(len(lens)), lens)
    doc = rng.integers(0, docs, len(word))
    order = np.lexsort((doc, word))
    c = cb.Corpus.from_arrays(np.concatenate([[0], np.cumsum(np.bincount(doc, minlength=docs))]),
                              np.concatenate([[0], np.cumsum(lens)]), doc[order].astype(np.int32))
    got = {}
    for item_tokens in (0, 40, 300):
        with cb.LDA(c, k, 0.1, 0.01, seed=4, item_tokens=item_tokens) as m:
            if proposal:
                with cb.Encoder(c.num_words, k, max_batch=128, seed=2) as enc:
                    m.set_proposal(enc)
            for steps in (1, 2, 5):
                z = m.mh_snapshot(3, steps)
                assert z.max() < k and (steps == 1 or (z != m.topics()).any())
                assert np.array_equal(z, got.setdefault(steps, z))
            m.iterate_mh(2, 3)
            assert np.array_equal(m.topics(), got.setdefault("chain", m.topics()))
