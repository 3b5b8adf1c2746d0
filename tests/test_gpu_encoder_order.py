"""The order in which the embedding gradient is summed.

The batch's (word, row) pairs are sorted by word, rows ascending inside a word,
and cut into chunks of 32; a word's terms are added one after the other inside a
chunk and the chunks' partial sums into zero.  With at most two chunks per word
that sum has one value, whatever order the GPU works in, and the batch (under
512 rows, so that no weight gradient is split) gives every run the same dX0.  So
the comparison is of bits: there is no tolerance.

Every document holds one word of its own, whose gradient row is dX0[b] / L_b;
with L_b a power of two that recovers dX0[b] exactly, and the other words'
gradients can be restated on the host in FP32."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import culda_cgs_b200 as cb
from culda_cgs_b200 import _ffi
from oracle import encoder_oracle as EO

pytestmark = pytest.mark.gpu

CHUNK = 32


def _batch(rng, docs, common):
    """Documents of 2^n tokens: the document's own word (id common + b) and common
    words, none of which occurs more than CHUNK + 1 times."""
    lens = 2 ** rng.integers(0, 6, docs)
    pool = rng.permutation(np.repeat(np.arange(common), CHUNK + 1))
    rest = lens - 1
    assert rest.sum() <= len(pool)
    words, at = [], 0
    for b, n in enumerate(rest):
        words.append(np.sort(np.append(pool[at:at + n], common + b)))
        at += n
    return np.concatenate([[0], np.cumsum(lens)]), np.concatenate(words), lens


def _restate(doc_ptr, words, lens, dx0, num_words):
    """dE in FP32, summed in the order the module describes."""
    row = np.repeat(np.arange(len(lens)), lens)
    order = np.argsort(words, kind="stable")
    grad = np.zeros((num_words, dx0.shape[1]), dtype=np.float32)
    for c0 in range(0, len(order), CHUNK):
        part, last = None, -1
        for t in list(order[c0:c0 + CHUNK]) + [None]:
            w = -2 if t is None else int(words[t])
            if w != last:
                if part is not None:
                    grad[last] = grad[last] + part
                part, last = np.zeros(dx0.shape[1], dtype=np.float32), w
            if t is not None:
                b = row[t]
                part = part + dx0[b] * np.float32(1.0 / lens[b])  # exact products: L_b is a power of two
    return grad


@pytest.mark.parametrize("docs,common", [(128, 60), (300, 200), (2, 4)])
def test_embedding_gradient_is_summed_in_row_order(docs, common):
    import torch

    rng = np.random.default_rng(docs)
    K, V = 128, common + docs
    doc_ptr, words, lens = _batch(rng, docs, common)
    with cb.Encoder(V, K, max_batch=docs) as enc:
        for n, v in EO.random_tensors(rng, V, K).items():
            enc.set(n, v)
        d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
             (doc_ptr.astype(np.int64), words.astype(np.int32), EO.random_target(rng, docs, K).astype(np.float32))]
        loss, runs = C.c_double(), []
        for _ in range(6):
            assert cb.lib().culda_encoder_backward(enc.handle, docs, None, *[C.c_void_p(x.data_ptr()) for x in d],
                                                   C.byref(loss), None) == 0
            runs.append(enc.get("E", grad=True).reshape(V, -1).copy())
    dx0 = runs[0][common:] * lens[:, None].astype(np.float32)
    want = _restate(doc_ptr, words, lens, dx0, V)
    for got in runs:
        assert np.array_equal(got, want)


def test_batch_of_too_many_tokens_is_refused():
    """Document numbers may repeat: 65536 times one document of 40,000 tokens is more
    than the sort's 32-bit positions hold.  The loss of the next pass is not touched."""
    import torch

    batch, n, V, K = 65536, 40_000, 50, 128
    with cb.Encoder(V, K, max_batch=batch) as enc:
        ptr = torch.tensor([0, n, n + 3], device="cuda")
        words = torch.arange(n + 3, device="cuda", dtype=torch.int32) % V
        target = torch.full((batch, K), 1.0 / K, device="cuda")
        loss, want = C.c_double(), C.c_double()

        def backward(docs, out):
            return cb.lib().culda_encoder_backward(enc.handle, len(docs), *[C.c_void_p(x.data_ptr()) for x in
                                                   (docs, ptr, words, target)], C.byref(out), None)

        short = torch.ones(4, device="cuda", dtype=torch.int32)
        assert backward(short, want) == 0
        many = torch.zeros(batch, device="cuda", dtype=torch.int32)
        assert backward(many, loss) == _ffi.CULDA_ERR_UNSUPPORTED
        assert backward(short, loss) == 0 and loss.value == want.value
