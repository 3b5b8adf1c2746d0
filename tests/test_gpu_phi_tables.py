"""culda_update_phi and culda_compute_phi_head against numpy: word lengths
around the kernel's limits (a warp's words, whole-CTA words from 2048 tokens,
words cut between CTAs from 8192 tokens, empty words), table rows of every
16-byte remainder.  Counts are exact; phi_head is one IEEE single division per
element, so it is exact too."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import culda_cgs_b200 as cb

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 31, 32, 33, 129, 0, 0, 2047, 2048, 2049, 8191, 8192, 8193, 0, 60_000, 5]


@pytest.mark.parametrize("k,shift", [(32, 0), (96, 1), (1024, 0), (1024, 3), (2080, 0), (4096, 2)])
def test_update_phi_and_phi_head(k, shift):
    import torch

    rng = np.random.default_rng(k + shift)
    # short words between the edge cases, one word of most of the tokens, many one-token and empty words
    lens = np.concatenate([LENGTHS, rng.integers(0, 90, 700), [300_000], rng.integers(0, 2, 3000), LENGTHS])
    v, n = len(lens), int(lens.sum())
    word_ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    z = (rng.integers(0, k, n) * rng.integers(0, 2, n)).astype(np.uint16)  # half the tokens on topic 0
    want = np.bincount(np.repeat(np.arange(v), lens) * k + z, minlength=v * k).reshape(v, k)
    d_ptr = torch.from_numpy(word_ptr).cuda()
    d_z = torch.from_numpy(z.view(np.int16)).cuda()
    phi = torch.full((v * k + 8,), -1, dtype=torch.int32, device="cuda")
    nk = torch.full((k,), -1, dtype=torch.int32, device="cuda")
    out = torch.full((v * k + 8,), -1.0, device="cuda")

    def at(t):
        return C.c_void_p(t.data_ptr() + 4 * shift)

    beta = np.float32(0.01)
    for _ in range(2):  # the second call starts from used tables
        assert cb.lib().culda_update_phi(k, v, d_ptr.data_ptr(), d_z.data_ptr(), at(phi), nk.data_ptr(), None) == 0
        assert cb.lib().culda_compute_phi_head(k, beta, v, at(phi), nk.data_ptr(), at(out), None) == 0
        got = phi.cpu().numpy()
        assert (got[:shift] == -1).all() and (got[shift + v * k:] == -1).all()
        assert np.array_equal(got[shift:shift + v * k].reshape(v, k), want)
        assert np.array_equal(nk.cpu().numpy(), want.sum(0))
        head = out.cpu().numpy()
        assert (head[:shift] == -1).all() and (head[shift + v * k:] == -1).all()
        den = want.sum(0).astype(np.float32) + np.float32(beta * np.float32(v))
        assert np.array_equal(head[shift:shift + v * k].reshape(v, k), (want.astype(np.float32) + beta) / den)


@pytest.mark.parametrize("k", [4096])
def test_tables_in_a_captured_stream(k):
    """The two entry points can be captured into a graph, at any K."""
    import torch

    rng = np.random.default_rng(1)
    lens = rng.integers(0, 40, 200)
    v, n = len(lens), int(lens.sum())
    z = rng.integers(0, k, n).astype(np.uint16)
    d_ptr = torch.from_numpy(np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)).cuda()
    d_z = torch.from_numpy(z.view(np.int16)).cuda()
    phi, head = torch.zeros(v, k, dtype=torch.int32, device="cuda"), torch.zeros(v, k, device="cuda")
    nk = torch.zeros(k, dtype=torch.int32, device="cuda")
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        assert cb.lib().culda_update_phi(k, v, d_ptr.data_ptr(), d_z.data_ptr(), phi.data_ptr(), nk.data_ptr(),
                                         s.cuda_stream) == 0
        assert cb.lib().culda_compute_phi_head(k, 0.01, v, phi.data_ptr(), nk.data_ptr(), head.data_ptr(),
                                               s.cuda_stream) == 0
    g.replay()
    torch.cuda.synchronize()
    want = np.bincount(np.repeat(np.arange(v), lens) * k + z, minlength=v * k).reshape(v, k)
    assert np.array_equal(phi.cpu().numpy(), want) and np.array_equal(nk.cpu().numpy(), want.sum(0))
    assert (head.cpu().numpy() > 0).all()
