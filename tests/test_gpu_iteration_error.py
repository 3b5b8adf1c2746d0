"""A device error ends a call of several iterations with the iteration that reports
it, although others are queued behind it.  The error is planted from the host, in
the context's error word between two calls (a few lines compiled against the
context's own header find it), so no kernel does anything wrong; every iteration
reports the word until it is cleared.  Topics, counts and iteration numbers are
compared with those of an undisturbed chain."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

import culda_cgs_b200 as cb
from culda_cgs_b200 import _ffi, build
from culda_cgs_b200.configs import TINY

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "context.h"
extern "C" __attribute__((visibility("default"))) int set_error_word(culda_ctx *ctx, int value) {
    return (int)cudaMemcpy(ctx->d_error, &value, sizeof value, cudaMemcpyHostToDevice);
}
"""


@pytest.fixture(scope="module")
def set_error_word(tmp_path_factory):
    src = tmp_path_factory.mktemp("error") / "e.cu"
    src.write_text(SOURCE)
    lib = src.with_suffix(".so")
    subprocess.run([build._nvcc(), "-std=c++17", *build.ARCH, "-shared", "-Xcompiler", "-fPIC", "-I", str(build.CSRC),
                    "-o", str(lib), str(src)], check=True)
    fn = C.CDLL(str(lib)).set_error_word
    fn.argtypes = [C.c_void_p, C.c_int]
    return lambda lda, value: fn(lda._ctx, value) == 0


def _state(lda):
    a, ja, _, cur = lda.theta()
    phi, nk = lda.phi()
    return lda.next_iteration, lda.topics(), a, ja, cur, phi, nk, lda.loglik_joint()


def _equal(x, y):
    return all(np.array_equal(a, b) for a, b in zip(x, y))


@pytest.mark.parametrize("flags", [0, _ffi.CULDA_FLAG_NO_GRAPH])
@pytest.mark.parametrize("mh", [False, True])
def test_the_call_ends_with_the_failing_iteration(set_error_word, mh, flags):
    corpus, k = cb.Corpus.generate(TINY.gen), TINY.k

    def run(lda, n):
        stats = (_ffi.IterStats * n)()
        fn = cb.lib().culda_iterate_mh if mh else cb.lib().culda_iterate
        rc = fn(lda._ctx, n, *([2] if mh else []), stats)
        return rc, [(s.iteration, s.status) for s in stats]

    with cb.LDA(corpus, k, TINY.alpha, TINY.beta, seed=5, flags=flags) as ref, \
            cb.LDA(corpus, k, TINY.alpha, TINY.beta, seed=5, flags=flags) as m:
        assert run(ref, 2)[0] == 0 and run(m, 2)[0] == 0
        for n in (1, 2, 5, 9):
            assert set_error_word(m, 1)
            rc, stats = run(m, n)
            assert rc == _ffi.CULDA_ERR_DEVICE_STATE
            first = ref.next_iteration
            assert stats == [(first, 1)] + [(0, 0)] * (n - 1)  # the later ones are not filled
            assert set_error_word(m, 0)
            assert run(ref, 1)[0] == 0
            assert _equal(_state(m), _state(ref))
        # and goes on from there
        assert run(ref, 6) == run(m, 6)
        assert _equal(_state(m), _state(ref))
