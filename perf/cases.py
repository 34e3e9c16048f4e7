"""What the framework is timed on: the work its users have it do, through its public entry points, over the range of
sizes that this repository's configurations, tests and benchmark name.

Six kinds of work, each with ranges of its own (`draw`) and one to four listed members:

  train    opt_gqa_cuda with gradients: the attention of one layer in a training step
  prefill  opt_gqa_cuda without gradients: the attention of one layer while a prompt is read; with `cache` the layer's
           K and V also go into a paged cache, as a serving program does before it decodes
  decode   PreparedDecode.step under its CUDA graph: one token for each running request
  eager    PagedKVCache.append_and_attend: a few tokens per request without a prepared plan
  merge    merge_forward_cuda: the standalone merge, for callers that hold the two branches themselves
  session  FullQwen2Session.step: one token of a whole randomly initialised model

`prepare` makes what a user's program holds before the call (inputs, cache contents, plan, model), `run` is one pass.
"""
import math
import os
import random
import sys

import torch

_PACKAGE = os.path.join(os.getcwd(), "moba-merge-cuda_b200")
for _p in (_PACKAGE, os.path.join(_PACKAGE, "examples")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

from moba_opt import PagedKVCache, run_impl  # noqa: E402
from moba_opt.ops.merge_cuda import merge_forward_cuda  # noqa: E402

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}

# Head shapes (query heads / KV heads) that the configurations and tests use.
_HEADS = ((8, 8), (8, 2), (14, 2), (12, 2), (28, 4), (32, 8), (4, 1), (6, 1))

# A pass of a drawn training case costs at most about this many attention operations (the long shard below has 1.8 times that).
_MOST_FLOPS = 2.0e13


def listed():
    return [
        # one request, the sparse attention layer of a small chat model: what a token's latency is made of
        dict(name="decode_one", kind="decode", requests=1, lo=16384, hi=16384, hq=14, hkv=2, dim=64, page=16, chunk=512,
             topk=4, mode="moba", dtype="bf16"),
        # a small batch on the dense layers of a model that mixes dense and sparse ones
        dict(name="decode_dense_8", kind="decode", requests=8, lo=16384, hi=32768, hq=28, hkv=4, dim=128, page=16, chunk=512,
             topk=4, mode="dense", dtype="fp16"),
        # the serving configuration: 64 requests with long contexts, page size not dividing the chunk
        dict(name="decode_64", kind="decode", requests=64, lo=4096, hi=65536, hq=12, hkv=2, dim=128, page=48, chunk=2048,
             topk=4, mode="moba", dtype="bf16"),
        # four new tokens for each of eight requests through the eager call (a verified draft, a short user turn)
        dict(name="eager_8x4", kind="eager", requests=8, tokens=4, lo=500, hi=8000, hq=14, hkv=2, dim=64, page=16, chunk=512,
             topk=4, dtype="bf16"),
        # the smallest prefill of the configurations: 2048 tokens, as many KV heads as query heads
        dict(name="prefill_2k", kind="prefill", seqs=1, tokens=2048, hq=8, hkv=8, dim=64, chunk=256, topk=3, dtype="bf16",
             precision="upstream", fused=False, cache=False),
        # a long prompt of a serving program: fused q/k/v projection in, attention out, K and V handed to the cache
        dict(name="prompt_64k", kind="prefill", seqs=1, tokens=65536, hq=14, hkv=2, dim=64, chunk=2048, topk=4, dtype="bf16",
             precision="upstream", fused=True, cache=True),
        # fine-tuning on a small packed batch with odd sequence lengths, half precision
        dict(name="train_ragged_6k", kind="train", seqs=3, tokens=6131, hq=8, hkv=2, dim=64, chunk=500, topk=3, dtype="fp16",
             precision="fp32", fused=False, deterministic=False),
        # an ordinary training batch at head dimension 128, many small chunks
        dict(name="train_d128_32k", kind="train", seqs=4, tokens=32768, hq=12, hkv=2, dim=128, chunk=512, topk=8, dtype="bf16",
             precision="upstream", fused=True, deterministic=False),
        # the headline configuration: four sequences of 32768 tokens
        dict(name="train_4x32k", kind="train", seqs=4, tokens=131072, hq=14, hkv=2, dim=64, chunk=2048, topk=3, dtype="bf16",
             precision="upstream", fused=False, deterministic=False),
        # one KV-head group of the long-context configuration: the largest case
        dict(name="train_128k", kind="train", seqs=1, tokens=131072, hq=4, hkv=1, dim=128, chunk=4096, topk=12, dtype="bf16",
             precision="upstream", fused=False, deterministic=False),
        # the merge of a 16384-token batch whose rows have up to three remote contributions
        dict(name="merge_16k", kind="merge", tokens=16384, heads=14, dim=64, kmax=3, dtype="bf16"),
        # one token of a small chat model in a short conversation, every other layer sparse; a third of the model's 24
        # layers, because on random weights rounding differences grow with depth until outputs cannot be compared
        dict(name="session_8", kind="session", layers=8, prompt=2000, hidden=896, hq=14, hkv=2, ffn=4864, vocab=151936,
             page=16, chunk=512, topk=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("train", "train", "train", "prefill", "prefill", "decode", "decode", "decode", "eager", "merge", "session"))
    hq, hkv = rng.choice(_HEADS)
    dim = rng.choice((64, 64, 64, 128, 128, 128, 96, 32))
    dtype = rng.choice(("bf16", "bf16", "bf16", "fp16"))
    if kind in ("train", "prefill"):
        while True:
            tokens = _log(rng, 1000, 131072)
            c = dict(kind=kind, seqs=rng.choice((1, 1, 2, 3, 4)), tokens=tokens, hq=hq, hkv=hkv, dim=dim,
                     chunk=rng.choice((256, 512, 500, 1024, 2048, 2048, 4096)), topk=rng.choice((2, 3, 3, 4, 4, 8, 12)), dtype=dtype,
                     precision=rng.choice(("upstream", "upstream", "fp32")), fused=rng.random() < 0.5)
            if kind == "train":
                c["deterministic"] = rng.random() < 0.2
            else:
                c["cache"] = rng.random() < 0.5
            # the cost bound, and partial rows of the remote branch that fit the card beside two other states
            if _attention_flops(c, 14) <= _MOST_FLOPS and tokens * hq * (c["topk"] - 1) * dim <= 1.2e9:
                return c
    if kind == "decode":
        dense = rng.random() < 0.25                   # dense layers matter where contexts are long
        hi = _log(rng, 16384 if dense else 2000, 65536)
        requests = _log(rng, 1, max(1, min(64, int(1.2e9 / (hi * hkv * dim)))))   # K and V of all requests: about 5 GB at most
        chunk = rng.choice((128, 512, 512, 1024, 2048))
        return dict(kind=kind, requests=requests, lo=hi // (2 if dense else rng.choice((1, 4, 16))), hi=hi, hq=hq, hkv=hkv, dim=dim,
                    page=rng.choice((16, 16, 48, 64)), chunk=chunk, topk=rng.choice((2, 4, 4, 8)), mode="dense" if dense else "moba",
                    dtype=dtype)
    if kind == "eager":
        hi = _log(rng, 1000, 32768)
        tokens = _log(rng, 1, 16)
        return dict(kind=kind, requests=_log(rng, 1, min(32, 64 // tokens)), tokens=tokens, lo=hi // 8, hi=hi, hq=hq, hkv=hkv, dim=dim,
                    page=rng.choice((16, 48, 64)), chunk=rng.choice((128, 512, 1024)), topk=rng.choice((2, 4, 8)), dtype=dtype)
    if kind == "merge":
        return dict(kind=kind, tokens=_log(rng, 500, 65536), heads=hq, dim=dim, kmax=rng.choice((1, 2, 3, 3, 7)), dtype=dtype)
    # prompts of at most topk chunks: on random weights a near tie between chunks is settled by rounding
    return dict(kind=kind, layers=rng.choice((2, 4, 6, 8)), prompt=rng.randint(500, 2040), hidden=896, hq=14, hkv=2, ffn=4864, vocab=151936,
                page=16, chunk=512, topk=4)


# ------------------------------------------------------------------------------------------------- sizes of a case
def _lengths(total, n):
    """`n` sequence lengths that add up to `total`: equal ones where they divide it, otherwise uneven and odd."""
    if n == 1 or total % n == 0:
        return [total // n] * n
    rng = random.Random(total * 31 + n)
    weight = [rng.uniform(0.3, 1.0) for _ in range(n)]
    got = [max(1, int(total * w / sum(weight))) for w in weight]
    got[-1] += total - sum(got)
    return got


def _contexts(c):
    """Cached tokens of every request: uniform between lo and hi, the same ones whatever the seed of the data."""
    rng = random.Random(c["lo"] * 131 + c["hi"] * 17 + c["requests"])
    return [rng.randint(c["lo"], c["hi"]) for _ in range(c["requests"])]


def _attended_pairs(lens, chunk, topk):
    total = 0
    for length in lens:
        n = -(-length // chunk)
        for i in range(n):
            size = chunk if i < n - 1 else length - (n - 1) * chunk
            total += size * (size + 1) // 2 + size * min(topk - 1, i) * chunk
    return total


def _attention_flops(c, per):
    return float(per) * c["dim"] * _attended_pairs(_lengths(c["tokens"], c["seqs"]), c["chunk"], c["topk"]) * c["hq"]


def _cached_tokens_read(length, chunk, topk, group):
    """Tokens of one KV head that a group of query heads reads for one token at position length - 1: the own chunk so
    far, and as many different earlier chunks as independent choices of the heads are expected to name."""
    cur = (length - 1) // chunk
    own = length - cur * chunk
    picks = min(topk - 1, cur)
    return own + (cur * (1.0 - (1.0 - picks / cur) ** group) * chunk if cur else 0.0)


def work(case):
    c = case
    kind = c["kind"]
    if kind in ("train", "prefill"):
        row = 2 * c["dim"] * c["tokens"]
        if kind == "train":       # q, k, v, dO in; out, dq, dk, dv out
            return {"bytes": row * (4 * c["hq"] + 4 * c["hkv"]), "flops": _attention_flops(c, 14)}
        stored = 2 * c["hkv"] if c["cache"] else 0
        return {"bytes": row * (2 * c["hq"] + 2 * c["hkv"] + stored), "flops": _attention_flops(c, 4)}
    if kind in ("decode", "eager"):
        group = c["hq"] // c["hkv"]
        tokens = read = 0
        for n in _contexts(c):
            for t in range(c.get("tokens", 1)):
                tokens += 1
                dense = c.get("mode") == "dense" or c["topk"] == 1
                read += (n + t + 1) if dense else _cached_tokens_read(n + t + 1, c["chunk"], c["topk"], group)
        if kind == "eager":       # the new tokens of a request share what they read
            read /= c["tokens"]
        return {"bytes": 4 * c["dim"] * c["hkv"] * read + 4 * c["dim"] * tokens * (c["hq"] + c["hkv"]),
                "flops": 4.0 * c["dim"] * c["hq"] * read}
    if kind == "merge":
        rows = c["tokens"] * c["heads"]
        return {"bytes": rows * (2 + c["kmax"]) * (2 * c["dim"] + 4) + rows * c["kmax"] * 8, "flops": 2.0 * rows * (1 + c["kmax"]) * c["dim"]}
    dim, h = c["hidden"] // c["hq"], c["hidden"]
    layer = h * (c["hq"] + 2 * c["hkv"]) * dim + h * c["hq"] * dim + 3 * h * c["ffn"]
    weights = c["layers"] * layer + c["vocab"] * h
    sparse = c["layers"] // 2
    read = sparse * _cached_tokens_read(c["prompt"] + 1, c["chunk"], c["topk"], c["hq"] // c["hkv"]) + (c["layers"] - sparse) * (c["prompt"] + 1)
    return {"bytes": 2 * weights + 4 * dim * c["hkv"] * read, "flops": 2.0 * weights + 4.0 * dim * c["hq"] * read}


def tolerance(case):
    kind = case["kind"]
    if kind == "merge":
        return {"rel": 4e-3} if case["dtype"] == "bf16" else {"rel": 1e-3}
    if kind == "session":
        return {"rel": 3e-2}
    if kind in ("decode", "eager"):
        return {"rel": 1e-2, "differ": 2e-3} if case["dtype"] == "bf16" else {"rel": 1.2e-3, "differ": 2e-3}
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 1.2e-3}


# ------------------------------------------------------------------------------------------------- one pass of each kind
def _normal(gen, *shape, dtype):
    return torch.randn(*shape, device="cuda", generator=gen).to(dtype)


def _qkv(c, gen, tokens):
    """q, k, v of one layer; `fused`: views of one projection's output, as a model with a fused q/k/v projection has them."""
    dtype, hq, hkv, dim = _DTYPES[c["dtype"]], c["hq"], c["hkv"], c["dim"]
    if c["fused"]:
        qkv = torch.empty(tokens, hq + 2 * hkv, dim, device="cuda", dtype=dtype)
        for h in range(hq + 2 * hkv):
            qkv[:, h] = torch.randn(tokens, dim, device="cuda", generator=gen)
        return qkv[:, :hq], qkv[:, hq:hq + hkv], qkv[:, hq + hkv:]
    return tuple(_normal(gen, tokens, h, dim, dtype=dtype) for h in (hq, hkv, hkv))


def _prefill_state(c, gen):
    lens = _lengths(c["tokens"], c["seqs"])
    offsets = [0]
    for n in lens:
        offsets.append(offsets[-1] + n)
    config = dict(chunk_size=c["chunk"], topk=c["topk"], route_precision=c["precision"])
    s = dict(kind=c["kind"], cu=torch.tensor(offsets, dtype=torch.int32, device="cuda"), longest=max(lens), config=config)
    q, k, v = _qkv(c, gen, c["tokens"])
    if c["kind"] == "train":
        config["deterministic_backward"] = c["deterministic"]
        s["d_out"] = _normal(gen, *q.shape, dtype=q.dtype)
        q, k, v = (t.detach().requires_grad_() for t in (q, k, v))
    elif c["cache"]:
        page = 16
        s["ids"], s["offsets"] = list(range(len(lens))), offsets
        s["cache"] = PagedKVCache(len(lens), max(lens) + 1024, c["hkv"], c["dim"], page_size=page,
                                  num_pages=sum(-(-n // page) for n in lens), chunk_size=c["chunk"], dtype=q.dtype)
        s["cache"].k_cache.zero_()
        s["cache"].v_cache.zero_()
    s["q"], s["k"], s["v"] = q, k, v
    return s


def _run_train(s):
    out = run_impl("opt_gqa_cuda", s["q"], s["k"], s["v"], s["cu"], s["longest"], s["config"])
    dq, dk, dv = torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["d_out"])
    return {"out": out, "dq": dq, "dk": dk, "dv": dv}


def _run_prefill(s):
    with torch.no_grad():
        cache = s.get("cache")
        if cache is None:
            return run_impl("opt_gqa_cuda", s["q"], s["k"], s["v"], s["cu"], s["longest"], s["config"])
        cache.reset()             # the slots of finished requests
        cache.append_prefill(s["k"], s["v"], sequence_ids=s["ids"], cu_seqlens=s["offsets"], check_finite=False)
        out = run_impl("opt_gqa_cuda", s["q"], s["k"], s["v"], s["cu"], s["longest"], s["config"])
        return {"out": out, "k_cache": cache.k_cache, "v_cache": cache.v_cache}


def _filled_cache(c, gen, room):
    """A cache with the requests' contexts, appended in rounds as running requests do, so that their pages are scattered."""
    lens, dtype = _contexts(c), _DTYPES[c["dtype"]]
    page = c["page"]
    cache = PagedKVCache(len(lens), max(lens) + room, c["hkv"], c["dim"], page_size=page,
                         num_pages=sum(-(-(n + room) // page) for n in lens), chunk_size=c["chunk"], dtype=dtype)
    step = max(512, max(lens) // 16)
    done = [0] * len(lens)
    while True:
        ids = [i for i, n in enumerate(lens) if done[i] < n]
        if not ids:
            return cache
        counts = [min(step, lens[i] - done[i]) for i in ids]
        cu = [0]
        for i, n in zip(ids, counts):
            done[i] += n
            cu.append(cu[-1] + n)
        k, v = (_normal(gen, cu[-1], c["hkv"], c["dim"], dtype=dtype) for _ in range(2))
        cache.append_prefill(k, v, sequence_ids=ids, cu_seqlens=cu, check_finite=False)


def _decode_state(c, gen):
    requests, dtype = c["requests"], _DTYPES[c["dtype"]]
    # room for as many steps as a timing of this case may take
    cache = _filled_cache(c, gen, 32768 if requests <= 4 else 16384)
    plan = cache.prepare_decode(list(range(requests)), c["hq"], topk=c["topk"], mode=c["mode"], check_finite=False)
    plan.capture("step")
    turns = [tuple(_normal(gen, requests, h, c["dim"], dtype=dtype) for h in (c["hq"], c["hkv"], c["hkv"])) for _ in range(4)]
    return dict(kind="decode", cache=cache, plan=plan, turns=turns, at=0)


def _run_decode(s):
    q, k, v = s["turns"][s["at"] % 4]
    s["at"] += 1
    r = s["plan"].step(q, k, v, use_graph=True)
    return {"output": r.output, "lse": r.lse, "selected": r.selected_blocks}


def _eager_state(c, gen):
    requests, tokens, dtype = c["requests"], c["tokens"], _DTYPES[c["dtype"]]
    cache = _filled_cache(c, gen, 4096 * tokens)   # room for as many passes as a timing may take
    turns = [tuple(_normal(gen, requests * tokens, h, c["dim"], dtype=dtype) for h in (c["hq"], c["hkv"], c["hkv"])) for _ in range(4)]
    return dict(kind="eager", cache=cache, turns=turns, at=0, ids=list(range(requests)), cu=[i * tokens for i in range(requests + 1)],
                topk=c["topk"])


def _run_eager(s):
    q, k, v = s["turns"][s["at"] % 4]
    s["at"] += 1
    r = s["cache"].append_and_attend(q, k, v, sequence_ids=s["ids"], cu_seqlens=s["cu"], topk=s["topk"])
    return {"output": r.output, "lse": r.lse, "selected": r.selected_blocks}


def _merge_state(c, gen):
    dtype, rows = _DTYPES[c["dtype"]], c["tokens"] * c["heads"]
    # contributions as a routed forward leaves them: per earlier chunk the rows in order, about a tenth of the slots unused
    mapping = torch.cat([(torch.rand(rows, device="cuda", generator=gen) < 0.9).nonzero()[:, 0] for _ in range(c["kmax"])])
    m = mapping.numel()
    return dict(kind="merge", kmax=c["kmax"], mapping=mapping,
                self_out=_normal(gen, c["tokens"], c["heads"], c["dim"], dtype=dtype),
                self_lse=torch.randn(c["tokens"], c["heads"], device="cuda", generator=gen) + 6.0,
                remote_out=_normal(gen, m, 1, c["dim"], dtype=dtype), remote_lse=torch.randn(m, device="cuda", generator=gen) + 6.0)


def _run_merge(s):
    return merge_forward_cuda(s["self_out"], s["self_lse"], s["remote_out"], s["remote_lse"], s["mapping"], kmax=s["kmax"],
                              check_capacity=False)


def _session_state(c, seed):
    from full_qwen2 import FullQwen2Session, random_qwen2
    room = 8192                   # steps that a timing may take
    model = random_qwen2(hidden=c["hidden"], layers=c["layers"], heads=c["hq"], kv_heads=c["hkv"], ffn=c["ffn"], vocab=c["vocab"],
                         max_positions=c["prompt"] + room, seed=seed)
    gen = torch.Generator().manual_seed(seed)
    ids = torch.randint(0, c["vocab"], (1, c["prompt"]), generator=gen).cuda()
    session = FullQwen2Session(model, c["prompt"] + room, mode="moba", chunk=c["chunk"], topk=c["topk"], page=c["page"],
                               backend="model_graph", dense_layers=range(0, c["layers"], 2))
    session.prefill(ids)
    session.prepare()
    return dict(kind="session", session=session, tokens=torch.randint(0, c["vocab"], (64,), generator=gen).tolist(), at=0)


def _run_session(s):
    token = s["tokens"][s["at"] % 64]
    s["at"] += 1
    return s["session"].step(token)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind in ("train", "prefill"):
        return _prefill_state(case, gen)
    if kind == "session":
        return _session_state(case, seed)
    return {"decode": _decode_state, "eager": _eager_state, "merge": _merge_state}[kind](case, gen)


def run(state):
    return {"train": _run_train, "prefill": _run_prefill, "decode": _run_decode, "eager": _run_eager, "merge": _run_merge,
            "session": _run_session}[state["kind"]](state)
