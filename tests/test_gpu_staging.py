"""Topics to and from pageable and pinned host arrays whose sizes straddle the
staging limits (2 MB slots, eight of them; staged from 16 MB on), from several threads at once,
and after the idle staging memory was handed back.  Copies are exact."""
from __future__ import annotations

import ctypes as C
import threading

import numpy as np
import pytest

import culda_cgs_b200 as cb

pytestmark = pytest.mark.gpu

STAGED = (16 << 20) // 2  # tokens of the smallest staged copy


def chain(n, k=32, seed=3):
    rng = np.random.default_rng(n)
    docs, words = max(2, n // 500), max(2, n // 800)
    word_ptr = np.linspace(0, n, words + 1).astype(np.int64)
    key = np.repeat(np.arange(words), np.diff(word_ptr)) * docs + rng.integers(0, docs, n)
    ids = (np.sort(key) % docs).astype(np.int32)
    doc_ptr = np.concatenate([[0], np.cumsum(np.bincount(ids, minlength=docs))])
    return cb.LDA(cb.Corpus.from_arrays(doc_ptr, word_ptr, ids), k, 0.5, 0.01, seed=seed), rng


@pytest.mark.parametrize("n", [STAGED - 1, STAGED, 5 * STAGED // 2 + 7])
def test_round_trip(n):
    import torch

    m, rng = chain(n)
    with m:
        z = rng.integers(0, m.k, n).astype(np.uint16)
        m.set_topics(z)
        assert np.array_equal(m.topics(), z)
        assert cb.lib().culda_trim_memory(0) == 0
        pinned = torch.empty(n, dtype=torch.int16, pin_memory=True)
        assert cb.lib().culda_get_topics(m._ctx, C.cast(pinned.data_ptr(), C.POINTER(C.c_uint16))) == 0
        assert np.array_equal(pinned.numpy().view(np.uint16), z)
        odd = np.empty(2 * n + 1, dtype=np.uint8)[1:]  # an odd address
        assert cb.lib().culda_get_topics(m._ctx, C.cast(odd.ctypes.data, C.POINTER(C.c_uint16))) == 0
        assert np.array_equal(odd.view(np.uint8), z.view(np.uint8))


def test_threads_copy_at_once():
    chains = [chain(STAGED + i, seed=i) for i in range(3)]
    failed = []

    def work(m, rng):
        for _ in range(2):
            z = rng.integers(0, m.k, m.num_tokens).astype(np.uint16)
            m.set_topics(z)
            if not np.array_equal(m.topics(), z):
                failed.append(m)

    threads = [threading.Thread(target=work, args=c) for c in chains]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for m, _ in chains:
        m.close()
    assert not failed
