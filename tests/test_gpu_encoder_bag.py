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
