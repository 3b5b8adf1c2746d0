"""The array of the segments' docs is optional: without it (no room for it at
set-up) the sampler finds the docs itself, with the same draws; and a token adds no
more to the context's block than the arrays that need it."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

import culda_cgs_b200 as cb
from culda_cgs_b200 import build
from culda_cgs_b200.configs import MINI

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "context.h"
extern "C" __attribute__((visibility("default"))) void *swap_segment_docs(culda_ctx *ctx, void *docs) {
    void *old = ctx->d_seg_doc;
    ctx->d_seg_doc = static_cast<int32_t *>(docs);
    return old;
}
"""


@pytest.fixture(scope="module")
def swap_segment_docs(tmp_path_factory):
    src = tmp_path_factory.mktemp("segments") / "s.cu"
    src.write_text(SOURCE)
    lib = src.with_suffix(".so")
    subprocess.run([build._nvcc(), "-std=c++17", *build.ARCH, "-shared", "-Xcompiler", "-fPIC", "-I", str(build.CSRC),
                    "-o", str(lib), str(src)], check=True)
    fn = C.CDLL(str(lib)).swap_segment_docs
    fn.argtypes, fn.restype = [C.c_void_p, C.c_void_p], C.c_void_p
    return fn


@pytest.mark.parametrize("k", [64, 1024])
def test_the_draws_without_the_array(swap_segment_docs, k):
    corpus = cb.Corpus.generate(MINI.gen)
    runs = []
    for without in (False, True):
        with cb.LDA(corpus, k, 50.0 / k, 0.01, seed=9) as m:
            docs = None
            if without:
                docs = swap_segment_docs(m._ctx, None)
                assert docs
                m.set_frozen_phi(None, None)  # captures the iteration again
            st = m.iterate(3)
            runs.append((m.topics(), [s["loglik"] for s in st], m.sample_snapshot(7)))
            if without:
                swap_segment_docs(m._ctx, docs)
    (z, ll, snap), (z2, ll2, snap2) = runs
    assert np.array_equal(z, z2) and ll == ll2
    assert np.array_equal(snap[0], snap2[0]) and snap[1] == snap2[1]


def test_bytes_per_token():
    """Documents that repeat one word: a segment is up to 32 tokens, so the segments' docs are few."""
    size = []
    docs = 60
    for length in (20_000, 40_000):
        n = docs * length
        corpus = cb.Corpus.from_arrays(np.arange(docs + 1, dtype=np.int64) * length, np.array([0, n], dtype=np.int64),
                                       np.repeat(np.arange(docs, dtype=np.int32), length))
        with cb.LDA(corpus, 64, 0.5, 0.01, seed=1) as m:
            m.iterate(1)
            size.append(m.info()["device_bytes"])
    # doc ids, token index, doc tokens, segment starts, uniforms: 4 bytes each; three topic arrays: 2 each
    assert (size[1] - size[0]) / (docs * 20_000) < 5 * 4 + 3 * 2 + 1
