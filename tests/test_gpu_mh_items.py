"""A Metropolis-Hastings pass draws the same topics however the words are cut
into work items: by a CTA (256 tokens or more), by a warp, split over items (the
hot rows), with the proposal's block table within one 128-byte line (K <= 1024)
or past it, and with an odd number of steps.  Draws are exact."""
from __future__ import annotations

import numpy as np
import pytest

import culda_cgs_b200 as cb
from test_gpu_parity import snapshot_of

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


@pytest.mark.parametrize("steps", [2, 5])
def test_pass_over_tables_past_the_l2(steps):
    """100,000 documents at K = 1024: 0.6 GB of proposal and n_dk tables, more than four times the L2, where a pass
    takes fewer CTAs and one of more than two steps keeps what it read of a token's topic.  The oracle's draws,
    but for decisions within 1e-6 of their boundary."""
    k, docs, seed = 1024, 100_000, 6
    rng = np.random.default_rng(9)
    word, doc = rng.integers(0, 700, 4 * docs), rng.permutation(np.repeat(np.arange(docs), 4))
    order = np.lexsort((doc, word))
    c = cb.Corpus.from_arrays(np.arange(docs + 1) * 4,
                              np.concatenate([[0], np.cumsum(np.bincount(word, minlength=700))]),
                              doc[order].astype(np.int32))
    with cb.LDA(c, k, 50.0 / k, 0.01, seed=seed) as m, cb.Encoder(c.num_words, k, 1024, seed=3) as enc:
        m.iterate(1)
        m.set_proposal(enc)
        got = m.mh_snapshot(5, steps=steps)
        want, margin = snapshot_of(m, c).mh(seed, 5, steps, cdf=m.proposal())
    assert np.array_equal(got[margin >= 1e-6], want[margin >= 1e-6]) and (got != want).mean() < 1e-3
