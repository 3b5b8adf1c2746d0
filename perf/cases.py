"""Workloads of the sampler and of its document encoder, as a user's program
runs them through the public entry points.

Every case is a dict of plain values.  `prepare` makes what a program holds
before the call (a corpus, a context, an encoder, a kernel-level work list),
`run` makes one pass, `work` says what a pass cannot do without, and `exact`
gives the computed numbers in 64 bits where they have such a value.

Corpora are synthetic: Zipf(1.05)-like word ranks, documents that mix a few
of 512 generating topics, lengths Poisson-like ("even"), lognormal ("mixed")
or Pareto ("uneven"), the laws of culda_cgs_b200/configs.py.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import culda_cgs_b200 as cb
from culda_cgs_b200 import _ffi
from culda_cgs_b200._ffi import check
from culda_cgs_b200.encoder import TENSORS, Encoder

BETA = 0.01
GEN_TOPICS = 512
MAX_LEN = {"even": 1000, "mixed": 5000, "uneven": 50_000}


def listed():
    return [
        # a chain on a toy corpus, stepped one iteration at a time as the reference's driver loop does:
        # latency and launches are all there is
        {"name": "train-tiny", "kind": "train", "docs": 200, "mean_len": 40, "law": "even", "vocab": 500, "k": 64,
         "iterations": 1},
        # the 1M-token configuration between two checkpoints of its topics
        {"name": "train-small", "kind": "train", "docs": 10_000, "mean_len": 100, "law": "even", "vocab": 20_000,
         "k": 1024, "iterations": 10},
        # the 60M-token headline configuration between two checkpoints
        {"name": "train-scale", "kind": "train", "docs": 300_000, "mean_len": 204, "law": "mixed", "vocab": 100_000,
         "k": 1024, "iterations": 10},
        # very uneven documents and a long vocabulary tail at a large K
        {"name": "train-uneven", "kind": "train", "docs": 400_000, "mean_len": 60, "law": "uneven",
         "vocab": 1_000_000, "k": 2048, "iterations": 3},
        # odd sizes and a K that is no power of two
        {"name": "train-ragged", "kind": "train", "docs": 37_311, "mean_len": 187, "law": "mixed", "vocab": 51_003,
         "k": 288, "iterations": 4},
        # new documents sampled against a trained model's fixed counts
        {"name": "foldin", "kind": "foldin", "docs": 50_000, "mean_len": 100, "law": "even", "vocab": 20_000,
         "k": 1024, "iterations": 4},
        # Metropolis-Hastings iterations, document and encoder proposals in turn
        {"name": "mh", "kind": "mh", "docs": 30_001, "mean_len": 200, "law": "mixed", "vocab": 40_000, "k": 512,
         "iterations": 4, "steps": 2, "proposal": True},
        # the joint log-likelihood a user tracks during training
        {"name": "evaluate", "kind": "evaluate", "docs": 60_000, "mean_len": 204, "law": "mixed", "vocab": 100_000,
         "k": 1024},
        # a whole job from host arrays: set-up, ten iterations, the topics back on the host
        {"name": "job", "kind": "job", "docs": 60_000, "mean_len": 204, "law": "mixed", "vocab": 100_000, "k": 1024,
         "iterations": 10},
        # an iteration through the kernel-level entry points, call by call as in the reference's driver
        {"name": "kernels", "kind": "kernels", "docs": 20_000, "mean_len": 204, "law": "mixed", "vocab": 50_000,
         "k": 1024},
        # topic distributions of a batch of documents from the encoder
        {"name": "encoder-infer", "kind": "infer", "docs": 8_000, "mean_len": 204, "law": "mixed", "vocab": 50_000,
         "k": 1024, "batch": 4000},
        # encoder training: eight steps, then the weights are read back
        {"name": "encoder-train", "kind": "fit", "docs": 8_192, "mean_len": 100, "law": "even", "vocab": 20_000,
         "k": 1024, "batch": 1024, "steps": 8},
    ]


def draw(rng):
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["train", "train", "train", "foldin", "mh", "evaluate", "job", "kernels", "infer", "fit"])
    law = rng.choice(["even", "mixed", "uneven"])
    c = {"kind": kind, "docs": log_int(150, 60_000), "mean_len": log_int(30, 300), "law": law,
         "vocab": log_int(400, 300_000), "k": 32 * log_int(1, 64)}
    if kind in ("train", "foldin", "job"):
        c["iterations"] = rng.randint(1, 5) if kind != "job" else rng.randint(3, 10)
    if kind in ("foldin", "kernels", "evaluate"):
        c["vocab"] = log_int(400, 60_000)
    if kind == "foldin":
        c["k"] = 32 * log_int(1, 32)
    if kind == "mh":
        c.update(vocab=log_int(400, 60_000), k=128 * rng.randint(1, 8), iterations=rng.randint(1, 4),
                 steps=rng.randint(1, 4), proposal=rng.random() < 0.7)
    if kind in ("infer", "fit"):
        c.update(docs=log_int(150, 8_192), vocab=log_int(400, 60_000), k=128 * rng.randint(1, 16))
        c["batch"] = rng.randint(max(1, c["docs"] // 8), c["docs"])
        if kind == "fit":
            c["steps"] = rng.randint(1, 8)
    return c


# ------------------------------------------------------------------ corpora
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _mix(x):
    """Elementwise 31-bit hash of int64 values."""
    x = (x * 0x2C1B3C6D + 0x297A2D39) & 0x7FFFFFFF
    x = ((x ^ (x >> 15)) * 0x45D9F3B) & 0x7FFFFFFF
    x = ((x ^ (x >> 13)) * 0x119DE1F3) & 0x7FFFFFFF
    return x ^ (x >> 16)


def _lengths(case):
    """The law's quantiles, so that a case's corpora have one token count whatever the seed."""
    d, mean, law = case["docs"], float(case["mean_len"]), case["law"]
    q = (torch.arange(d, device="cuda", dtype=torch.float64) + 0.5) / d
    normal = math.sqrt(2.0) * torch.erfinv(2.0 * q - 1.0)
    if law == "even":
        x = mean + math.sqrt(mean) * normal
    elif law == "mixed":
        x = torch.exp(math.log(mean) - 0.32 + 0.8 * normal)
    else:
        x = mean / 3 * (1.0 - q) ** (-1 / 1.5)
    return x.round().long().clamp(1, MAX_LEN[law])


def _words(case):
    """Distinct words: the vocabulary, or a quarter of the tokens where that is less."""
    return max(1, min(case["vocab"], int(_lengths(case).sum()) // 4))


def _tokens(case, seed):
    """(doc lengths, doc of every token, word of every token, generating topic), doc by doc; every word occurs."""
    gen = _generator(seed)
    lens = _lengths(case)[torch.randperm(case["docs"], generator=gen, device="cuda")]
    doc = torch.repeat_interleave(torch.arange(case["docs"], device="cuda"), lens)
    n, words = doc.numel(), _words(case)
    # the document's j-th topic, j geometric
    j = torch.log2(1.0 - torch.rand(n, generator=gen, device="cuda")).neg().div(0.5).long().clamp_(max=15)
    topic = _mix(_mix(doc + seed * 7919) + j) % GEN_TOPICS
    # word rank r with density ~ 1/r^1.05 on [1, words], then within r's octave [2^m, 2^(m+1)) a stretch of an
    # eighth of the octave that depends on the topic
    u = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
    s = -0.05
    rank = (1.0 + u * (float(words) ** s - 1.0)) ** (1.0 / s)
    m = torch.log2(rank).floor().clamp_(0, 40)
    size = torch.exp2(m).long()
    at = (rank.long() - size).clamp_(min=0) // 8
    word = (size - 1 + (_mix(topic * 64 + m.long()) + at) % size) % words
    word[torch.randperm(n, generator=gen, device="cuda")[:words]] = torch.arange(words, device="cuda")
    return lens, doc, word, topic


def _ptr(counts):
    return torch.cat([counts.new_zeros(1), counts.cumsum(0)])


def _corpus(case, seed):
    """The word-major corpus on the host and the tokens' generating topics in its order (on the GPU)."""
    lens, doc, word, topic = _tokens(case, seed)
    order = torch.sort(word * case["docs"] + doc, stable=True)[1]
    words = _words(case)
    word_ptr = _ptr(torch.bincount(word, minlength=words))
    corpus = cb.Corpus.from_arrays(_ptr(lens).cpu().numpy(), word_ptr.cpu().numpy(),
                                   doc[order].int().cpu().numpy())
    return corpus, topic[order]


def _alpha(case):
    return 50.0 / case["k"]


def _lda(case, seed, corpus):
    return cb.LDA(corpus, case["k"], _alpha(case), BETA, seed=seed + 1)


def _topics(case, topic, seed):
    """Topics of a chain in progress: three quarters of the tokens on their generating topic."""
    z = _mix(topic) % case["k"]
    noise = torch.randint(0, case["k"], z.shape, generator=_generator(seed + 5), device="cuda")
    keep = torch.rand(z.shape, generator=_generator(seed + 6), device="cuda") < 0.75
    return torch.where(keep, z, noise)


def _u16(z):
    return z.to(torch.int16).cpu().numpy().view(np.uint16)


# ------------------------------------------------------------------ encoder
WIDTH, HIDDEN = _ffi.CULDA_ENC_EMBED, _ffi.CULDA_ENC_HIDDEN


def _weights(case, words, seed):
    gen = _generator(seed + 11)

    def normal(*shape, scale):
        return scale * torch.randn(*shape, generator=gen, device="cuda")

    k = case["k"]
    return {"E": normal(words, WIDTH, scale=0.3), "W1": normal(HIDDEN, WIDTH, scale=0.08),
            "b1": normal(HIDDEN, scale=0.1), "W2": normal(HIDDEN, HIDDEN, scale=0.06),
            "b2": normal(HIDDEN, scale=0.1), "W3": normal(k, HIDDEN, scale=0.06), "b3": normal(k, scale=0.1)}


def _bag(case, seed):
    """Documents as a CSR of word ids (words ascending inside a document) and the batches' document numbers."""
    lens, doc, word, _ = _tokens(case, seed)
    words = _words(case)
    order = torch.sort(doc * words + word, stable=True)[1]
    steps = case.get("steps", 1)
    gen = _generator(seed + 12)
    docs = [torch.randperm(case["docs"], generator=gen, device="cuda")[:case["batch"]].int() for _ in range(steps)]
    return _ptr(lens), word[order].int(), words, docs


def _encoder(case, words, weights, batch):
    enc = Encoder(words, case["k"], max_batch=batch, seed=1, lr=1e-3)
    for name, value in weights.items():
        enc.set(name, value.cpu().numpy())
    return enc


def _targets(case, seed):
    gen = _generator(seed + 13)
    return [torch.softmax(3 * torch.randn(case["batch"], case["k"], generator=gen, device="cuda"), 1)
            for _ in range(case["steps"])]


def _p(t):
    return C.c_void_p(t.data_ptr())


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("infer", "fit"):
        doc_ptr, words, num_words, docs = _bag(case, seed)
        enc = _encoder(case, num_words, _weights(case, num_words, seed), case["batch"])
        state = {"case": case, "enc": enc, "doc_ptr": doc_ptr, "words": words, "docs": docs}
        if kind == "infer":
            state["probs"] = torch.empty(case["batch"], case["k"], device="cuda")
        else:
            state["targets"] = _targets(case, seed)
            state["host"] = {n: torch.empty(enc.shape(n), pin_memory=True) for n in TENSORS}
        return state
    corpus, topic = _corpus(case, seed)
    state = {"case": case, "corpus": corpus, "seed": seed}
    if kind == "job":
        return state
    if kind == "kernels":
        state.update(_kernel_state(case, corpus, _topics(case, topic, seed)))
        state["seed"] = seed + 1
        return state
    state["lda"] = lda = _lda(case, seed, corpus)
    if kind == "evaluate":
        lda.set_topics(_u16(_topics(case, topic, seed)))
    elif kind == "foldin":
        # the trained model: counts of twice the documents over the same vocabulary
        k = case["k"]
        word = torch.repeat_interleave(torch.arange(corpus.num_words, device="cuda"),
                                       torch.from_numpy(np.diff(corpus.word_ptr)).cuda())
        phi = sum(torch.bincount(word * k + _topics(case, topic, seed + 20 + i), minlength=corpus.num_words * k)
                  for i in range(2)).view(-1, k)
        lda.set_frozen_phi(phi.int().cpu().numpy(), phi.sum(0).int().cpu().numpy())
    elif kind == "mh":
        lda.set_topics(_u16(_topics(case, topic, seed)))
        if case["proposal"]:
            with _encoder(case, corpus.num_words, _weights(case, corpus.num_words, seed), 1024) as enc:
                lda.set_proposal(enc)
    else:
        lda.iterate(8)  # a chain that has left its random start
    return state


def _kernel_state(case, corpus, z):
    """Device arrays and the work list for the kernel-level entry points."""
    lib, k = cb.lib(), case["k"]
    word_ptr, doc_ptr, ids = corpus.word_ptr, corpus.doc_ptr, corpus.doc_ids
    hot = C.c_int32()
    wp = word_ptr.ctypes.data_as(C.POINTER(C.c_int64))
    n = lib.culda_build_items(corpus.num_words, wp, 4096, None, 0, C.byref(hot))
    items = (_ffi.Item * n)()
    lib.culda_build_items(corpus.num_words, wp, 4096, items, n, C.byref(hot))
    ip = ids.ctypes.data_as(C.POINTER(C.c_int32))
    seg = np.zeros(len(ids), dtype=np.int32)
    nseg = lib.culda_build_segments(len(ids), ip, items, n, 32, seg.ctypes.data_as(C.POINTER(C.c_int32)), len(ids))
    listing = np.frombuffer(items, dtype=np.uint8).reshape(n, C.sizeof(_ffi.Item))
    split = listing[[i for i in range(n) if items[i].hot >= 0]]
    capacity = (np.minimum(np.diff(doc_ptr), k) + 31) // 32 * 32
    start = np.concatenate([[0], np.cumsum(capacity)])
    rows = np.stack([start[:-1], start[:-1]], 1).astype(np.int32)

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a)).cuda()

    s = {"items": dev(listing), "hot": dev(split) if len(split) else torch.zeros(64, dtype=torch.uint8, device="cuda"),
         "seg": dev(seg[:nseg]), "word_ptr": dev(word_ptr), "doc_ptr": dev(doc_ptr), "ids": dev(ids),
         "rows": dev(rows), "theta": torch.zeros(int(start[-1]), dtype=torch.int32, device="cuda"),
         "z": z.to(torch.int16), "num_items": n, "num_hot": hot.value, "num_hot_items": len(split)}
    s["doc_tok"] = torch.sort(s["ids"], stable=True)[1].int()
    s["z_out"] = torch.zeros_like(s["z"])
    s["phi"] = torch.zeros(corpus.num_words, k, dtype=torch.int32, device="cuda")
    s["phi_head"] = torch.zeros(corpus.num_words, k, device="cuda")
    s["nk"] = torch.zeros(k, dtype=torch.int32, device="cuda")
    s["ll"] = torch.zeros(1, dtype=torch.float64, device="cuda")
    s["err"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    s["ws"] = torch.zeros(max(lib.culda_sample_workspace(k, n, hot.value),
                              lib.culda_update_theta_workspace(k, corpus.num_docs)), dtype=torch.uint8, device="cuda")
    length = np.diff(doc_ptr).astype(np.float64)
    s["doc_term"] = float((length * np.log(length + k * float(np.float32(_alpha(case))))).sum())
    return s


# ---------------------------------------------------------------------- run
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("train", "foldin"):
        stats = state["lda"].iterate(case["iterations"])
        return {"topics": state["lda"].topics(), "loglik": [s["loglik"] for s in stats],
                "theta_nnz": [s["theta_nnz"] for s in stats]}
    if kind == "mh":
        stats = state["lda"].iterate_mh(case["iterations"], case["steps"])
        return {"topics": state["lda"].topics(), "accept_rate": [s["accept_rate"] for s in stats]}
    if kind == "evaluate":
        return {"loglik_joint": state["lda"].loglik_joint()}
    if kind == "job":
        with _lda(case, state["seed"], state["corpus"]) as lda:
            stats = lda.iterate(case["iterations"])
            return {"topics": lda.topics(), "loglik": [s["loglik"] for s in stats]}
    if kind == "kernels":
        return _run_kernels(state, case)
    lib, enc = cb.lib(), state["enc"]
    if kind == "infer":
        check(lib.culda_encoder_forward(enc.handle, case["batch"], _p(state["docs"][0]), _p(state["doc_ptr"]),
                                           _p(state["words"]), _p(state["probs"]), None))
        return {"probs": state["probs"]}
    losses = []
    for docs, target in zip(state["docs"], state["targets"]):
        loss = C.c_double()
        check(lib.culda_encoder_train_step(enc.handle, case["batch"], _p(docs), _p(state["doc_ptr"]),
                                              _p(state["words"]), _p(target), C.byref(loss), None))
        losses.append(loss.value)
    for name, which in TENSORS.items():
        check(lib.culda_encoder_get_tensor(enc.handle, which, _p(state["host"][name])))
    return {"loss": np.array(losses, dtype=np.float32), **state["host"]}


def _run_kernels(s, case):
    lib, corpus, k = cb.lib(), s["corpus"], case["k"]
    alpha = _alpha(case)
    check(lib.culda_update_phi(k, corpus.num_words, _p(s["word_ptr"]), _p(s["z"]), _p(s["phi"]), _p(s["nk"]), None))
    check(lib.culda_compute_phi_head(k, BETA, corpus.num_words, _p(s["phi"]), _p(s["nk"]), _p(s["phi_head"]), None))
    check(lib.culda_update_theta(k, corpus.num_docs, _p(s["doc_ptr"]), _p(s["doc_tok"]), _p(s["z"]), None,
                                    _p(s["rows"]), _p(s["theta"]), _p(s["nk"]), None, _p(s["ws"]), s["ws"].numel(),
                                    None))
    args = _ffi.SampleArgs(
        k=k, alpha=alpha, beta=BETA, num_docs=corpus.num_docs, num_words=corpus.num_words,
        num_tokens=corpus.num_tokens, word_ptr=_p(s["word_ptr"]), doc_ids=_p(s["ids"]), topics_in=_p(s["z"]),
        topics_out=_p(s["z_out"]), theta=_p(s["theta"]), theta_rows=_p(s["rows"]), nk=_p(s["nk"]),
        items=_p(s["items"]), seg_start=_p(s["seg"]), num_segs=s["seg"].numel(), num_items=s["num_items"],
        num_hot=s["num_hot"], hot_items=_p(s["hot"]), num_hot_items=s["num_hot_items"],
        theta_capacity=s["theta"].numel(), seed=s["seed"], iteration=3, group_lanes=_ffi.CULDA_SAMPLER_FLAT,
        loglik_sum=_p(s["ll"]), error=_p(s["err"]))
    check(lib.culda_sample(C.byref(args), _p(s["ws"]), s["ws"].numel(), None))
    ll = C.c_double()
    check(lib.culda_loglik(_p(s["ll"]), s["doc_term"], corpus.num_tokens, C.byref(ll), None))
    return {"phi": s["phi"], "phi_head": s["phi_head"], "theta": s["theta"], "rows": s["rows"], "nk": s["nk"],
            "topics": s["z_out"], "loglik": ll.value}


# --------------------------------------------------------------------- work
def work(case):
    kind, k = case["kind"], case["k"]
    n = float(case["docs"]) * case["mean_len"]
    # entries of a document's theta row, as a share of its tokens and no more than K
    row = min(float(k), 0.6 * case["mean_len"])
    theta = case["docs"] * row
    vocab = min(case["vocab"], n)
    if kind in ("train", "foldin", "job", "mh"):
        it = case["iterations"]
        fixed = 4 * vocab * k if kind == "foldin" else 0
        # per iteration: doc ids, topics in and out, theta read and written
        per = 8 * n + 8 * theta + fixed
        walk = case["steps"] * 4 if kind == "mh" else 2 * row
        return {"bytes": it * per + 2 * n + (8 * n if kind == "job" else 0), "flops": it * n * walk}
    if kind == "evaluate":
        return {"bytes": 2 * n + 4 * theta, "flops": 20 * (theta + min(n, vocab * k))}
    if kind == "kernels":
        return {"bytes": 8 * vocab * k + 16 * n + 8 * theta, "flops": 2 * n * row + 2 * vocab * k}
    b = case["batch"]
    mlp = WIDTH * HIDDEN + HIDDEN * HIDDEN + HIDDEN * k
    tokens = b * case["mean_len"]
    if kind == "infer":
        return {"bytes": 4 * tokens + 2 * min(vocab, tokens) * WIDTH + 2 * mlp + 4 * b * k,
                "flops": 2 * b * mlp + tokens * WIDTH}
    params = vocab * WIDTH + mlp
    # per step: bag rows in and out, the targets, Adam over every weight; then the weights to the host
    per = 4 * tokens + 4 * b * k + 28 * params
    return {"bytes": case["steps"] * per + 4 * params, "flops": case["steps"] * (6 * b * mlp + 3 * tokens * WIDTH)}


# -------------------------------------------------------------------- exact
def exact(case, seed):
    kind = case["kind"]
    if kind == "evaluate":
        return {"loglik_joint": _exact_joint(case, seed)}
    if kind == "kernels":
        return _exact_kernels(case, seed)
    if kind in ("infer", "fit"):
        return _exact_encoder(case, seed)
    return None  # a chain's topics are draws


def _word_doc(case, seed):
    lens, doc, word, topic = _tokens(case, seed)
    order = torch.sort(word * case["docs"] + doc, stable=True)[1]
    return lens, doc[order], word[order], _topics(case, topic[order], seed)


def _exact_joint(case, seed):
    lens, doc, word, z = _word_doc(case, seed)
    k, v, d = case["k"], _words(case), case["docs"]
    a, b = float(np.float32(_alpha(case))), float(np.float32(BETA))

    def lg(x):
        return torch.lgamma(x.double())

    def pairs(key, prior):
        counts = torch.unique(key, return_counts=True)[1]
        return (lg(counts + prior) - math.lgamma(prior)).sum()

    nk = torch.bincount(z, minlength=k)
    total = pairs(word * k + z, b) + pairs(doc * k + z, a)
    total += (math.lgamma(v * b) - lg(nk + v * b)).sum() + (math.lgamma(k * a) - lg(lens + k * a)).sum()
    return float(total)


def _exact_kernels(case, seed):
    lens, doc, word, z = _word_doc(case, seed)
    k, v, d = case["k"], _words(case), case["docs"]
    a, b = float(np.float32(_alpha(case))), float(np.float32(BETA))
    phi = torch.bincount(word * k + z, minlength=v * k).view(v, k).double()
    head = (phi + b) / (phi.sum(0) + v * b)
    theta = torch.bincount(doc * k + z, minlength=d * k).view(d, k).double() + a
    ll = 0.0
    for t in range(0, doc.numel(), 100_000):
        di, wi = doc[t:t + 100_000], word[t:t + 100_000]
        ll += float((torch.log((theta[di] * head[wi]).sum(1)) - torch.log(lens[di] + k * a)).sum())
    return {"phi": None, "phi_head": head, "theta": None, "rows": None, "nk": None, "topics": None,
            "loglik": ll / doc.numel()}


def _exact_encoder(case, seed):
    doc_ptr, words, num_words, docs = _bag(case, seed)
    w = {n: t.double().requires_grad_(True) for n, t in _weights(case, num_words, seed).items()}

    def log_q(batch):
        batch = batch.long()
        lens = doc_ptr[batch + 1] - doc_ptr[batch]
        row = torch.repeat_interleave(torch.arange(len(batch), device="cuda"), lens)
        first = torch.repeat_interleave(doc_ptr[batch] - _ptr(lens)[:-1], lens)
        tok = words[torch.arange(len(row), device="cuda") + first].long()
        x = torch.zeros(len(batch), WIDTH, dtype=torch.float64, device="cuda")
        x = x.index_add(0, row, w["E"][tok]) / lens[:, None]
        for i in "12":
            x = torch.nn.functional.gelu(x @ w["W" + i].T + w["b" + i])
        return torch.log_softmax(x @ w["W3"].T + w["b3"], 1)

    if case["kind"] == "infer":
        with torch.no_grad():
            return {"probs": log_q(docs[0]).exp()}
    mean = {n: torch.zeros_like(t) for n, t in w.items()}
    square = {n: torch.zeros_like(t) for n, t in w.items()}
    losses = []
    for step, (batch, target) in enumerate(zip(docs, _targets(case, seed)), 1):
        loss = -(target.double() * log_q(batch)).sum() / case["batch"]
        losses.append(float(loss))
        grads = torch.autograd.grad(loss, list(w.values()))
        with torch.no_grad():
            for (n, t), g in zip(w.items(), grads):
                mean[n] = 0.9 * mean[n] + 0.1 * g
                square[n] = 0.999 * square[n] + 0.001 * g * g
                t -= 1e-3 * (mean[n] / (1 - 0.9 ** step)) / (torch.sqrt(square[n] / (1 - 0.999 ** step)) + 1e-8)
    return {"loss": np.array(losses), **{n: t.detach() for n, t in w.items()}}
