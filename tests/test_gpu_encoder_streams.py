"""One encoder used on two streams, one call after the other: a call that returns the
loss has nothing of its own left on its stream, so the next call may run on another.
The loss is compared with that of the same passes on one stream (1e-6 relative:
the order of 8-row sums in FP32 terms added in FP64)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import culda_cgs_b200 as cb
from culda_cgs_b200 import _ffi
from oracle import encoder_oracle as EO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 300])
def test_losses_of_passes_on_alternating_streams(batch):
    import torch

    rng = np.random.default_rng(batch)
    V, K = 200, 128
    doc_ptr, words = EO.random_batch(rng, V, batch, 30)
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
         (doc_ptr.astype(np.int64), words.astype(np.int32), EO.random_target(rng, batch, K).astype(np.float32))]
    d_ptr, d_words, d_target = [C.c_void_p(x.data_ptr()) for x in d]
    bad = torch.full_like(d[1], V)
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    with cb.Encoder(V, K, max_batch=batch) as enc:
        loss = C.c_double()

        def backward(stream, words=d_words):
            return cb.lib().culda_encoder_backward(enc.handle, batch, None, d_ptr, words, d_target, C.byref(loss),
                                                   C.c_void_p(stream.cuda_stream))

        assert backward(streams[0]) == 0
        want = loss.value
        for i in range(40):
            s = streams[i % 2]
            assert backward(s) == 0
            assert s.query(), "the call has returned and its stream has work"
            assert abs(loss.value - want) <= 1e-6 * want
            # a failing call clears its error word, and the loss, before it returns
            if i % 4 == 3:
                assert backward(s, C.c_void_p(bad.data_ptr())) == _ffi.CULDA_ERR_DEVICE_STATE
                assert s.query()


def test_a_forward_pass_that_fails_leaves_no_error_behind():
    import torch

    rng = np.random.default_rng(4)
    V, K, batch = 200, 128, 5
    doc_ptr, words = EO.random_batch(rng, V, batch, 30)
    ptr, good = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
                 (doc_ptr.astype(np.int64), words.astype(np.int32)))
    bad = torch.full_like(good, V)
    probs = torch.zeros(batch, K, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    with cb.Encoder(V, K, max_batch=batch) as enc:
        for i in range(20):
            s = streams[i % 2]
            for w, rc in ((bad, _ffi.CULDA_ERR_DEVICE_STATE), (good, 0)):
                assert cb.lib().culda_encoder_forward(enc.handle, batch, None, *[C.c_void_p(x.data_ptr()) for x in
                                                      (ptr, w, probs)], C.c_void_p(s.cuda_stream)) == rc
                assert s.query()
