"""The encoder's embedding bag at the lengths where its pipeline can go wrong:
documents of no token, of fewer tokens than warps, around the ring's 12 rows and
the 32 word ids a warp holds, one much longer than the rest; and a word id out of
range.  q is compared with the FP64 oracle (2e-3 absolute, as in the other
encoder tests); the bag alone is checked through weights that pass the mean on."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import culda_cgs_b200 as cb
from culda_cgs_b200 import _ffi
from oracle import encoder_oracle as EO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 60])
def test_forward_at_the_bag_limits(batch):
    import torch

    rng = np.random.default_rng(batch)
    V, K = 400, 128
    lens = np.array([0, 1, 7, 8, 9, 31, 32, 33, 95, 96, 97, 8 * 12, 8 * 12 + 1, 8 * 32, 8 * 32 + 1, 5000] * 4)[:max(batch, 16)]
    lens = rng.permutation(lens)
    doc_ptr = np.concatenate([[0], np.cumsum(lens)])
    words = rng.integers(0, V, doc_ptr[-1])
    t = {k: v.astype(np.float32).astype(np.float64) for k, v in EO.random_tensors(rng, V, K).items()}
    with cb.Encoder(V, K, max_batch=batch) as enc:
        for k, v in t.items():
            enc.set(k, v)
        d_ptr = torch.from_numpy(doc_ptr.astype(np.int64)).cuda()
        d_words = torch.from_numpy(words.astype(np.int32)).cuda()
        probs = torch.zeros(batch, K, device="cuda")

        def forward():
            return cb.lib().culda_encoder_forward(enc.handle, batch, None, C.c_void_p(d_ptr.data_ptr()),
                                                  C.c_void_p(d_words.data_ptr()), C.c_void_p(probs.data_ptr()), None)

        assert forward() == 0
        ora = EO.EncoderOracle(t).run(doc_ptr, words, np.arange(batch), np.full((batch, K), 1.0 / K))
        assert np.abs(probs.cpu().numpy() - ora["q"]).max() < 2e-3
        d_words[int(doc_ptr[batch]) - 1] = V  # the last token of the last document with tokens
        assert forward() == _ffi.CULDA_ERR_DEVICE_STATE


BAG_LENGTHS = [1, 7, 8, 9, 31, 32, 33, 95, 96, 97, 8 * 12 + 1, 8 * 32 - 1, 8 * 32, 8 * 32 + 1, 8 * 96, 8 * 97, 5000]


@pytest.mark.parametrize("seed", [0, 1])
def test_the_bag_alone(seed):
    """The mean itself, bit for bit.  Word c's embedding is 1 in column c and in column
    255, so a column's sum is a whole number (a token left out or taken twice changes
    it) and column 255 of the mean is 1.  With one document in the batch
    dW1[h, c] = dP1[h] * mean[c], a product of two BF16 numbers, which FP32 holds
    exactly: the mean is dW1[h, c] / dW1[h, 255]."""
    import torch

    rng = np.random.default_rng(seed)
    V, K = 255, 128
    lens = np.array(BAG_LENGTHS)
    doc_ptr = np.concatenate([[0], np.cumsum(lens)])
    words = rng.integers(0, V, doc_ptr[-1])
    emb = np.zeros((V, 256))
    emb[np.arange(V), np.arange(V)] = emb[:, 255] = 1.0
    with cb.Encoder(V, K, max_batch=1, seed=3 + seed) as enc:
        enc.set("E", emb)
        d = [torch.from_numpy(x).cuda() for x in (doc_ptr.astype(np.int64), words.astype(np.int32))]
        target = torch.from_numpy(EO.random_target(rng, 1, K).astype(np.float32)).cuda()
        for i, n in enumerate(lens):
            which = torch.tensor([i], dtype=torch.int32, device="cuda")
            loss = C.c_double()
            assert cb.lib().culda_encoder_backward(enc.handle, 1, *[C.c_void_p(x.data_ptr()) for x in
                                                   (which, *d, target)], C.byref(loss), None) == 0
            g = enc.get("W1", grad=True)
            h = np.abs(g[:, 255]).argmax()
            count = np.bincount(words[doc_ptr[i]:doc_ptr[i + 1]], minlength=256)
            count[255] = n
            mean = torch.from_numpy(count.astype(np.float32) * (np.float32(1.0) / np.float32(n)))
            assert np.array_equal(g[h] / g[h, 255], mean.to(torch.bfloat16).float().numpy()), n


def _batch(rng, V, lens):
    """Documents of the given lengths, each with its words in order, so runs of one word occur."""
    doc_ptr = np.concatenate([[0], np.cumsum(lens)])
    words = np.concatenate([np.sort((V * rng.random(n) ** 3).astype(np.int64)) for n in lens] + [np.zeros(0, int)])
    return doc_ptr, words


def _grads(enc, batch, doc_ptr, words, target, fn):
    import torch

    d = [torch.from_numpy(a).cuda() for a in (doc_ptr.astype(np.int64), words.astype(np.int32), target.astype(np.float32))]
    loss = C.c_double()
    assert fn(enc.handle, batch, None, *[C.c_void_p(x.data_ptr()) for x in d], C.byref(loss), None) == 0
    return {n: enc.get(n, grad=True).astype(np.float64).ravel() for n in EO.NAMES}


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("lens", [[0, 1, 31, 32, 33, 64, 65, 2], [4096, 4097, 0, 20_000, 5], [4097]])
def test_embedding_gradient_at_the_length_limits(lens):
    """dE against the oracle (2e-2 relative Frobenius, as the other gradients):
    documents of one CTA, those its helpers share, runs of one word."""
    rng = np.random.default_rng(len(lens))
    V, K, batch = 300, 128, len(lens)
    doc_ptr, words = _batch(rng, V, lens)
    t = {k: v.astype(np.float32).astype(np.float64) for k, v in EO.random_tensors(rng, V, K).items()}
    target = EO.random_target(rng, batch, K).astype(np.float32).astype(np.float64)
    with cb.Encoder(V, K, max_batch=batch) as enc:
        for k, v in t.items():
            enc.set(k, v)
        got = _grads(enc, batch, doc_ptr, words, target, cb.lib().culda_encoder_backward)
        want = EO.EncoderOracle(t).run(doc_ptr, words, np.arange(batch), target)["grads"]
        for n in EO.NAMES:
            assert _rel(got[n], want[n].ravel()) < 2e-2, n


@pytest.mark.parametrize("V,K", [(37, 128), (1000, 640)])
def test_training_step_refreshes_every_copy(V, K):
    """After a step, an encoder given the same weights anew (whose BF16 copies and
    transposes come from the plain conversion) has the same forward pass bit for
    bit and the same gradients up to the order of FP32 sums (1e-5)."""
    import torch

    rng = np.random.default_rng(V)
    batch = 150
    doc_ptr, words = _batch(rng, V, rng.integers(1, 40, batch))
    target = EO.random_target(rng, batch, K)
    with cb.Encoder(V, K, max_batch=batch, lr=1e-2) as a, cb.Encoder(V, K, max_batch=batch) as b:
        before = a.get("W3")
        _grads(a, batch, doc_ptr, words, target, cb.lib().culda_encoder_train_step)
        assert (a.get("W3") != before).mean() > 0.9
        for n in EO.NAMES:
            b.set(n, a.get(n))
        probs = []
        for enc in (a, b):
            q = torch.zeros(batch, K, device="cuda")
            d = [torch.from_numpy(x).cuda() for x in (doc_ptr.astype(np.int64), words.astype(np.int32))]
            assert cb.lib().culda_encoder_forward(enc.handle, batch, None, *[C.c_void_p(x.data_ptr()) for x in d],
                                                  C.c_void_p(q.data_ptr()), None) == 0
            probs.append(q.cpu().numpy())
        assert np.array_equal(*probs)
        ga, gb = (_grads(e, batch, doc_ptr, words, target, cb.lib().culda_encoder_backward) for e in (a, b))
        for n in EO.NAMES:
            assert _rel(ga[n], gb[n]) < 1e-5, n
