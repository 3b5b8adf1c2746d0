"""A kernel's dynamic shared-memory limit belongs to the process, the sizes to the
topic count: contexts and calls of different K, one after the other and from two
threads, must not take each other's room away.  Results are compared with those
of the same calls alone, bit for bit."""
from __future__ import annotations

import ctypes as C
import threading

import numpy as np
import pytest

import culda_cgs_b200 as cb
from culda_cgs_b200.configs import TINY

pytestmark = pytest.mark.gpu


def _chain(k, between=lambda: None):
    """Topics and joint log-likelihood of a short chain against frozen counts, whose graphs are captured after `between`."""
    corpus = cb.Corpus.generate(TINY.gen)
    with cb.LDA(corpus, k, 50.0 / k, 0.01, seed=3, device=0) as m:
        m.iterate(1)
        phi, nk = m.phi()
        between()
        m.set_frozen_phi(phi, nk)  # captures the iteration again
        ll = [s["loglik"] for s in m.iterate(2)]
        return m.topics(), ll, m.loglik_joint()


def _same(a, b):
    return np.array_equal(a[0], b[0]) and a[1:] == b[1:]


@pytest.mark.parametrize("k,smaller", [(1024, 64), (4096, 2048), (4096, 32)])
def test_a_smaller_context_leaves_the_limit(k, smaller):
    want = _chain(k)
    assert _same(_chain(k, lambda: _chain(smaller)), want)


class _UpdatePhi:
    """culda_update_phi at one K on a stream of its own.  Nothing here waits for the whole
    device, which is not allowed while another thread captures."""

    def __init__(self, k):
        import torch

        n, v = 20_000, 50
        self.k, self.v, self.stream = k, v, torch.cuda.Stream()
        with torch.cuda.stream(self.stream):
            self.ptr = torch.arange(0, n + 1, n // v, dtype=torch.int64, device="cuda")
            self.z = (torch.arange(n, device="cuda") * 7 % k).to(torch.int16)
            self.out = [torch.zeros(v, k, dtype=torch.int32, device="cuda"),
                        torch.zeros(k, dtype=torch.int32, device="cuda")]
            self.host = [torch.empty_like(t, device="cpu").pin_memory() for t in self.out]
        self.stream.synchronize()

    def __call__(self):
        import torch

        tables = [C.c_void_p(t.data_ptr()) for t in (self.ptr, self.z, *self.out)]
        assert cb.lib().culda_update_phi(self.k, self.v, *tables, C.c_void_p(self.stream.cuda_stream)) == 0
        with torch.cuda.stream(self.stream):
            for h, d in zip(self.host, self.out):
                h.copy_(d, non_blocking=True)
        self.stream.synchronize()
        return [h.numpy().copy() for h in self.host]


def test_threads_of_different_k():
    sizes = (64, 2048, 4096)
    tables = {k: _UpdatePhi(k) for k in sizes}
    want = {k: (_chain(k), tables[k]()) for k in sizes}
    wrong = []

    def work(k):
        try:
            for _ in range(12):
                assert _same(_chain(k), want[k][0])
                for _ in range(20):
                    assert all(np.array_equal(a, b) for a, b in zip(tables[k](), want[k][1]))
        except BaseException as e:  # noqa: BLE001
            wrong.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
