"""The measured workloads: what programs that use this framework have it do.

Kinds of case, each through the public entry points (one pass = one ``run``):

  resident  one Gibbs iteration of a chain whose corpus stays on the device:
            ``Sampler.corpus_sweep`` (the headline benchmark's loop)
  stream    one iteration over one host buffer by the reference's protocol:
            ``sample_phi``, then ``sample_z_async`` / ``sync_buffer`` with
            pinned host arrays, topics copied back into them
  device    ``sample_phi`` and the allocation-free sweep of documents that the
            caller holds in device memory (``gpulda_sample_z_device_noalloc``)
  batch     iterations of many independent chains (``BatchChains``), their
            topics read back
  serve     fold-in of new documents against a fixed model (``serve.Server``):
            submit, drain, poll.  Launch mode: its kernels end with their
            batch, so a pass can be waited for

The corpora are LDA-generated like ``gpupolyaurnlda_b200.corpus``: topics
Dirichlet(0.01) times Zipf(1.05) word weights, documents Dirichlet(0.1), words
ranked by frequency.  The topics and the set of document lengths belong to the
case, the documents (and the order of their lengths) to the seed: states of one
case are different documents of one language, as the buffers of a streamed
corpus are, and have the same number of tokens.  ``start`` says where the chain stands:
"trained" passes continue from the generating topics (most of a run's
iterations), "random" passes draw the topics of uniformly labelled documents
(its first iterations).

The library holds one model and one resident corpus per process, so preparing
a state makes a new model, and states prepared earlier go on with it (the
resident kind: with its corpus as well).

Every result is an integer of a random chain (topics, counts), or follows
from such integers (theta, the log-likelihood): there is no value of it that
plain torch or numpy reaches without running the sampler, so ``exact`` has
none.
"""
from __future__ import annotations

import gc
import math

import numpy as np
import torch

import gpupolyaurnlda_b200 as g
from gpupolyaurnlda_b200 import batch, serve

ZIPF, TOPIC_CONC, DOC_CONC, BETA = 1.05, 0.01, 0.1, 0.01
N_BUFFERS = 4


def listed():
    return [
        # The smallest call: one iteration of a demo-sized chain (the small
        # workload), with the log-likelihood that a training loop reports.
        # Launches and latency count.
        dict(name="small_resident", kind="resident", K=20, V=5000, D=2000, mu=4.6, sigma=0.1, lo=1, hi=400,
             start="trained", loglik=True),
        # The headline workload at its full size: K=1000, 3e5 documents, 1e8 tokens.
        dict(name="mid_resident", kind="resident", K=1000, V=100000, D=300000, mu=5.5, sigma=0.8, lo=10, hi=5000,
             start="trained", loglik=False),
        # Many short documents (abstracts, messages) at K=1000.
        dict(name="short_docs_resident", kind="resident", K=1000, V=140000, D=400000, mu=4.2, sigma=0.6, lo=5, hi=2000,
             start="trained", loglik=False),
        # Ten thousand topics: the large-K store.
        dict(name="large_k_resident", kind="resident", K=10000, V=30000, D=300000, mu=4.2, sigma=0.6, lo=5, hi=2000,
             start="trained", loglik=False),
        # A small ragged corpus with an odd number of topics and long documents
        # (books, 1e3 to 6e4 tokens).
        dict(name="long_docs_resident", kind="resident", K=333, V=20011, D=1501, mu=8.0, sigma=0.9, lo=3, hi=60000,
             start="trained", loglik=True),
        # The reference's protocol on one host buffer of a streamed corpus.
        dict(name="mid_stream", kind="stream", K=1000, V=50000, D=50000, mu=5.5, sigma=0.8, lo=10, hi=5000,
             start="trained", loglik=False),
        # The same with a small buffer: copies and launches count.
        dict(name="small_stream", kind="stream", K=100, V=8003, D=1000, mu=5.0, sigma=1.0, lo=1, hi=5000,
             start="trained", loglik=False),
        # First iterations from random topics, documents in device memory.
        dict(name="random_start_device", kind="device", K=1000, V=50000, D=60000, mu=5.5, sigma=0.8, lo=10, hi=5000,
             start="random", loglik=False),
        # Large K with the documents in device memory.
        dict(name="large_k_device", kind="device", K=4096, V=20000, D=20000, mu=4.5, sigma=1.0, lo=1, hi=5000,
             start="trained", loglik=False),
        # Independent chains side by side (per-group topic models).
        dict(name="batch_16", kind="batch", problems=16, K=1000, V=20000, D=4000, mu=4.5, sigma=1.0, lo=1, hi=65535,
             iters=4),
        # Fold-in of a batch of new documents, and of a single one.
        dict(name="serve_6000", kind="serve", K=1000, V=50000, D=6000, mu=5.0, sigma=1.2, lo=5, hi=2000, iters=50),
        dict(name="serve_one", kind="serve", K=200, V=20000, D=1, mu=5.0, sigma=0.3, lo=50, hi=400, iters=50),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["resident", "resident", "stream", "device", "batch", "serve"])
    mu, sigma, lo = rng.uniform(3.5, 6.5), rng.uniform(0.2, 1.1), rng.choice([1, 5, 10])
    mean = math.exp(mu + sigma * sigma / 2)
    case = dict(kind=kind, mu=round(mu, 3), sigma=round(sigma, 3), lo=lo, hi=rng.choice([2000, 5000, 20000]))
    if kind == "batch":
        case.update(problems=rng.randint(2, 24), K=_log_uniform(rng, 30, 2048), V=_log_uniform(rng, 1000, 20000),
                    D=max(8, int(_log_uniform(rng, 20000, 600000) / mean)), iters=rng.randint(1, 6))
    elif kind == "serve":
        case.update(K=_log_uniform(rng, 16, 2048), V=_log_uniform(rng, 1000, 50000),
                    D=max(1, int(_log_uniform(rng, 200, 300000) / mean)), iters=rng.choice([20, 50, 100]))
    else:
        # up to 3e7 tokens and 3e8 (word, topic) cells
        K = _log_uniform(rng, 8, 12000)
        case.update(K=K, V=_log_uniform(rng, 500, min(140000, 300000000 // K)),
                    D=max(4, int(_log_uniform(rng, 100000, 30000000) / mean)),
                    start=rng.choice(["trained", "trained", "random"]), loglik=rng.random() < 0.25)
    return case


# --- inputs -------------------------------------------------------------------

_topic_cache = {"key": None}


def _topics(K, V):
    """The topics' cumulative word distributions, row k offset by k (float64 on
    the GPU), words ranked by their overall frequency.  They are the case's,
    not the seed's, and kept until another case wants others."""
    key = (K, V)
    if _topic_cache["key"] != key:
        _topic_cache.clear()
        gen = torch.Generator("cuda").manual_seed(1000003 * K + V)
        lg = torch._standard_gamma(torch.full((K, V), TOPIC_CONC + 1.0, dtype=torch.float64, device="cuda"),
                                   generator=gen).log_()
        lg += torch.rand((K, V), dtype=torch.float64, device="cuda", generator=gen).clamp_min_(1e-300).log_().div_(
            TOPIC_CONC)
        lg -= ZIPF * torch.arange(1, V + 1, dtype=torch.float64, device="cuda").log()[None, :]
        lg -= lg.amax(dim=1, keepdim=True)
        p = lg.exp_()
        p /= p.sum(dim=1, keepdim=True)
        p = p[:, torch.argsort(p.sum(dim=0), descending=True)]
        cdf = torch.cumsum(p, dim=1)
        del p, lg
        cdf /= cdf[:, -1:].clone()
        cdf += torch.arange(K, dtype=torch.float64, device="cuda")[:, None]
        _topic_cache.update(key=key, cdf=cdf.reshape(-1))
    return _topic_cache["cdf"]


def _lengths(case, D):
    gen = torch.Generator("cuda").manual_seed(D)
    L = torch.exp(case["mu"] + case["sigma"] * torch.randn(D, dtype=torch.float64, device="cuda", generator=gen))
    return L.round_().clamp_(case["lo"], case["hi"]).long()


def _documents(case, seed, K=None, V=None, D=None):
    """Lengths, words and generating topics of the seed's documents (int64, GPU)."""
    K, V, D = K or case["K"], V or case["V"], D or case["D"]
    L = _lengths(case, D)
    N = int(L.sum())
    gen = torch.Generator("cuda").manual_seed(seed)
    rand = lambda n: torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)
    L = L[torch.randperm(D, device="cuda", generator=gen)]
    first = torch.repeat_interleave(torch.cumsum(L, 0) - L, L)
    # Dirichlet-multinomial topics by their urn: token i of a document takes a
    # new uniform topic with probability c / (c + i), else the topic of an
    # earlier token, found by following the references to their roots
    c = DOC_CONC * K
    i = torch.arange(N, device="cuda") - first
    u = rand(N) * (c + i)
    ref = torch.where(u < c, torch.arange(N, device="cuda"), first + (u - c).long().clamp_min_(0).minimum(i - 1))
    del u, i, first
    while True:
        up = ref[ref]
        if torch.equal(up, ref):
            break
        ref = up
    z = torch.randint(0, K, (N,), device="cuda", generator=gen)[ref]
    del ref, up
    w = torch.searchsorted(_topics(K, V), z + rand(N), right=True).clamp_max_(K * V - 1) - z * V
    return L, w.clamp_(0, V - 1), z


def _host(t):
    return t.to(torch.int32).cpu().numpy().view(np.uint32)


def _pinned(t):
    out = torch.empty(t.shape, dtype=torch.int32, pin_memory=True)
    out.copy_(t)
    return out.numpy().view(np.uint32)


# --- states -------------------------------------------------------------------

_live = {}  # the process's model ("sampler", "counts") or server


def _release(keep_server=None):
    if keep_server is not None and _live.get("server_key") == keep_server:
        return
    for name in ("sampler", "server"):
        if name in _live:
            _live[name].close()
    _live.clear()
    gc.collect()


def _new_model(case, w, z, buffer_size, max_D):
    """A fresh model whose counts are those of the given tokens."""
    K, V = case["K"], case["V"]
    _release()
    torch.cuda.empty_cache()
    s = g.Sampler(50.0 / K, BETA, K, _host(torch.bincount(w, minlength=V)), buffer_size=buffer_size, max_D=max_D,
                  n_buffers=N_BUFFERS, seed=1, flags=g.GPULDA_FLAG_LOGLIK if case["loglik"] else 0)
    counts = s.count_table()
    counts.copy_(torch.bincount(w * K + z, minlength=K * V))
    torch.cuda.synchronize()
    _live.update(sampler=s, counts=counts)
    return s


def _start_topics(case, z, seed):
    if case["start"] == "trained":
        return z
    gen = torch.Generator("cuda").manual_seed(seed + 7919)
    return torch.randint(0, case["K"], z.shape, device="cuda", generator=gen)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed)
    if kind == "serve":
        return _prepare_serve(case, seed)
    L, w, z = _documents(case, seed)
    z = _start_topics(case, z, seed)
    N, D = len(w), len(L)
    state = {"case": case}
    if kind == "resident":
        s = _new_model(case, w, z, 16, 4)
        s.corpus_load(_host(z), _host(w), _host(L))
    elif kind == "stream":
        _new_model(case, w, z, N, D)
        state.update(slot=seed % N_BUFFERS, z=_pinned(z), w=_pinned(w), d=_pinned(L))
    else:
        _new_model(case, w, z, 16, 4)
        state.update(z=z.int(), w=w.int(), d=L.int(), stream=torch.cuda.Stream())
    torch.cuda.synchronize()
    return state


def _prepare_batch(case, seed):
    """Problems of different sizes around the case's, one chain each, taken
    through the first iterations."""
    _release()
    specs = []
    for p in range(case["problems"]):
        # a few different vocabularies and topic numbers, document numbers from 1/4 to 7/4
        K = max(8, case["K"] // (1, 5, 20)[p % 3])
        V = max(200, case["V"] // (1, 2)[p % 2])
        D = max(2, case["D"] * (1 + 2 * (p % 4)) // 4)
        L, w, z = _documents(case, 64 * seed + p, K, V, D)
        specs.append((K, V, L, w, z))
    problems = [batch.ProblemSpec(50.0 / K, BETA, K, _host(torch.bincount(w, minlength=V)), _host(z), _host(w),
                                  _host(L), seed=p, loglik=False) for p, (K, V, L, w, z) in enumerate(specs)]
    chains = batch.BatchChains(problems)
    chains.sweep(20)
    return {"case": case, "chains": chains}


def _prepare_serve(case, seed):
    """Requests of the seed; the server and its model are the case's."""
    K, V = case["K"], case["V"]
    key = (K, V, case["iters"])
    _release(keep_server=key)
    if "server" not in _live:
        # the model of a chain: Poisson counts of a training corpus of 200
        # tokens a word around the topics
        cdf = _topics(K, V).view(K, V)
        gen = torch.Generator("cuda").manual_seed(K + V)
        p = torch.diff(cdf - torch.arange(K, dtype=torch.float64, device="cuda")[:, None], dim=1,
                       prepend=torch.zeros((K, 1), dtype=torch.float64, device="cuda")).clamp_min_(0)
        x = torch.poisson(p * (200.0 * V / K), generator=gen)
        q = (x * (4294967296.0 / x.sum(dim=1, keepdim=True).clamp_min(1.0))).floor_().clamp_max_(4294967295.0)
        q = q.t().contiguous().long().cpu().numpy().astype(np.uint32)
        del p, x, cdf
        torch.cuda.empty_cache()
        _live["server"] = serve.Server(case["iters"], mode="launch", slots=32, q=q, K=K, alpha=50.0 / K, seed=1,
                                       pool_bytes=1 << 29)
        _live["server_key"] = key
    L, w, _ = _documents(case, seed)
    ids = np.arange(len(L), dtype=np.uint64)
    return {"case": case, "ids": ids, "lengths": _host(L), "words": _host(w)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        chains = state["chains"]
        chains.sweep(case["iters"])
        return [chains.z(p).view(np.int32) for p in range(chains.n)]
    if kind == "serve":
        server = _live["server"]
        server.submit(state["ids"], state["lengths"], state["words"])
        server.drain()
        r = server.poll(len(state["ids"]))
        at = np.empty(len(state["ids"]), np.int64)  # results come in the order they finished
        at[r["ids"].astype(np.int64)] = np.arange(len(at))
        return {"theta": r["theta"][at], "loglik": r["ll"][at], "skipped": r["skipped"][at].view(np.int32)}
    s, out = _live["sampler"], {"counts": _live["counts"]}
    if kind == "resident":
        s.corpus_sweep(1)
    elif kind == "stream":
        s.sample_phi()
        s.sweep_buffer(state["slot"], state["z"], state["w"], state["d"])
        out["z"] = state["z"].view(np.int32)
    else:
        s.sample_phi()
        with torch.cuda.stream(state["stream"]):
            # the first iteration takes the documents as they came; a trained
            # chain goes on from its last topics
            z = state["z"].clone() if case["start"] == "random" else state["z"]
            g.check(g.lib().gpulda_sample_z_device_noalloc(
                z.data_ptr(), state["w"].data_ptr(), state["d"].data_ptr(), len(state["d"]), len(z),
                state["stream"].cuda_stream), "sample_z_device_noalloc")
        out["z"] = z
    if case["loglik"]:
        out["loglik"], out["skipped"] = s.loglik()
    return out


def _mean_length(case):
    """Mean of round(lognormal) clipped to [lo, hi]."""
    n = 4096
    u = (np.arange(n) + 0.5) / n
    x = math.sqrt(2.0) * torch.erfinv(torch.from_numpy(2.0 * u - 1.0)).numpy()
    return float(np.clip(np.round(np.exp(case["mu"] + case["sigma"] * x)), case["lo"], case["hi"]).mean())


def work(case):
    """Bytes of one pass.  An iteration reads the counts and writes the new ones
    (8 bytes a cell), reads every token's word and topic and writes its topic
    (12), reads every document's length (4).  Serving reads the words and
    writes theta and the log-likelihood.  The gathers of Phi depend on the
    chain and are not in it."""
    K, V, N = case["K"], case["V"], case["D"] * _mean_length(case)
    if case["kind"] == "serve":
        return {"bytes": 4.0 * N + case["D"] * (4.0 * K + 12.0), "flops": 0}
    if case["kind"] == "batch":
        total = 0.0
        for p in range(case["problems"]):
            k, v = max(8, K // (1, 5, 20)[p % 3]), max(200, V // (1, 2)[p % 2])
            d = max(2, case["D"] * (1 + 2 * (p % 4)) // 4)
            total += 8.0 * k * v + 12.0 * N * d / case["D"] + 4.0 * d
        return {"bytes": case["iters"] * total, "flops": 0}
    return {"bytes": 8.0 * K * V + 12.0 * N + 4.0 * case["D"], "flops": 0}


def exact(case, seed):
    return None
