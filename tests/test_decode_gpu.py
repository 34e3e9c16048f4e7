"""GPU parity of the KV cache and decode path against the FP64 oracle.  The cases follow the
reference's decode tests (tests/test_paged_decode.py): cache read-back bit-equal to what was
appended, chunk means, legality and ranking of routes, output/LSE under the kernel's own routes
(bf16: atol = rtol = 0.02, rel-L2 < 0.01, LSE atol 5e-4), page sizes that do not divide the chunk,
recycled pages, chunked (multi-token) appends, per-head routing known answers, error atomicity."""
import numpy as np
import pytest
import torch

from helpers import (CLUSTER_8, CLUSTER_16, DECODE_GOLDENS, FIXED, FIXED_DEEP, STREAMED, attend_kernels, bits_to_torch, load, torch_to_f64,
                     two_threads)
from oracle import moba_oracle as mo

pytestmark = pytest.mark.gpu


def rand(shape, seed, dtype=torch.bfloat16):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to("cuda", dtype)


def assert_payload(cache, sid, k, v):
    got_k, got_v = cache.materialize(sid)
    assert torch.equal(got_k, k) and torch.equal(got_v, v)


def check(cache, result, q):
    import moba_opt.grouped_attention as ga
    ga.check_status()
    C = cache.chunk_size
    keys, values = [], []
    for sid in range(len(cache.lengths)):
        k, v = cache.materialize(sid)
        keys.append(torch_to_f64(k))
        values.append(torch_to_f64(v))
        closed = cache.lengths[sid] // C
        if closed:
            half = cache.dtype == torch.float16
            want = mo.chunk_means(keys[-1], C, rounding=mo.fp16_round if half else mo.bf16_round)
            got = torch_to_f64(cache._means[sid, :closed])
            np.testing.assert_allclose(got, want, atol=1e-5, rtol=0.002 if half else 0.01)   # at most one ulp of the format apart
    qf = torch_to_f64(q)
    if result.selected_blocks is not None:
        route = result.selected_blocks.cpu().numpy()
        for row, (sid, pos) in enumerate(zip(result.sequence_ids, result.positions)):
            history = pos // C
            assert (route[row, :, 0] == history).all()
            means = torch_to_f64(cache._means[sid, :history]) if history else None
            for head in range(q.shape[1]):
                chosen = [int(c) for c in route[row, head, 1:] if c >= 0]
                assert len(chosen) == min(history, route.shape[-1] - 1)
                assert len(set(chosen)) == len(chosen) and all(c < history for c in chosen)
                if not chosen or len(chosen) == history:
                    continue
                kvh = head // (q.shape[1] // cache.num_kv_heads)
                scores = means[:, kvh] @ qf[row, head]
                rest = [i for i in range(history) if i not in chosen]
                bound = max(1e-6, float((np.abs(means[:, kvh]) @ np.abs(qf[row, head])).max())
                            * 4 * np.finfo(np.float32).eps * cache.head_dim)
                assert scores[chosen].min() + bound >= scores[rest].max()
    sel = None if result.selected_blocks is None else result.selected_blocks.cpu().numpy()
    want, lse = mo.decode_attend(qf, keys, values, result.sequence_ids, result.positions, C, sel)
    out = torch_to_f64(result.output)
    assert np.isfinite(out).all() and bool(torch.isfinite(result.lse).all())
    np.testing.assert_allclose(out, want, atol=0.02, rtol=0.02)
    assert np.linalg.norm(out - want) / max(np.linalg.norm(want), 1e-8) < 0.01
    np.testing.assert_allclose(torch_to_f64(result.lse), lse, atol=5e-4, rtol=2e-5)


@pytest.mark.parametrize("name", DECODE_GOLDENS)
def test_decode_matches_reference_golden(name):
    """Same inputs and hand-made routes as the fixtures produced by reference/decode_reference.py."""
    from moba_opt import PagedKVCache
    g = load(name)
    lengths, hq, hkv, dim, chunk = g["lengths"], int(g["hq"]), int(g["hkv"]), int(g["dim"]), int(g["chunk"])
    n = len(lengths)
    ks = [bits_to_torch(g[f"k{i}"], "cuda") for i in range(n)]
    vs = [bits_to_torch(g[f"v{i}"], "cuda") for i in range(n)]
    cache = PagedKVCache(n, int(max(lengths)) + 1, hkv, dim, page_size=5, chunk_size=chunk, dtype=ks[0].dtype)
    cache.append(torch.cat(ks), torch.cat(vs), sequence_ids=list(range(n)), cu_seqlens=[0] + [int(x) for x in np.cumsum(lengths)])
    q = bits_to_torch(g["q"], "cuda")
    dense = cache.attend(q, sequence_ids=list(range(n)), mode="dense")
    np.testing.assert_allclose(torch_to_f64(dense.output), g["out_dense"], atol=0.02, rtol=0.02)
    np.testing.assert_allclose(torch_to_f64(dense.lse), g["lse_dense"], atol=5e-4, rtol=2e-5)
    check(cache, dense, q)
    check(cache, cache.attend(q, sequence_ids=list(range(n)), topk=int(g["topk"])), q)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("kind", ["paged", "contiguous"])
@pytest.mark.parametrize("hq,hk", [(1, 1), (8, 1), (8, 2), (28, 4), (32, 8)])
def test_incremental_decode(kind, hq, hk, dtype):
    from moba_opt import ContiguousKVCache, PagedKVCache
    from functools import partial
    rand = partial(globals()["rand"], dtype=dtype)
    cache = (PagedKVCache(2, 32, hk, 64, chunk_size=4, page_size=3, dtype=dtype) if kind == "paged"
             else ContiguousKVCache(2, 32, hk, 64, chunk_size=4, dtype=dtype))
    k, v = rand((9, hk, 64), 101), rand((9, hk, 64), 102)
    cache.append(k, v, sequence_ids=[0, 1], cu_seqlens=[0, 4, 9])
    stored_k, stored_v = [k[:4], k[4:]], [v[:4], v[4:]]
    for sid in range(2):
        assert_payload(cache, sid, stored_k[sid], stored_v[sid])
    for step in range(3):
        q, k, v = rand((2, hq, 64), 103 + step), rand((2, hk, 64), 113 + step), rand((2, hk, 64), 123 + step)
        result = cache.append_and_attend(q, k, v, sequence_ids=[0, 1], topk=2)
        for sid in range(2):
            stored_k[sid] = torch.cat((stored_k[sid], k[sid:sid + 1]))
            stored_v[sid] = torch.cat((stored_v[sid], v[sid:sid + 1]))
            assert_payload(cache, sid, stored_k[sid], stored_v[sid])
        check(cache, result, q)
        check(cache, cache.attend(q, sequence_ids=[0, 1], mode="dense"), q)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("dim", [8, 16, 24, 40, 64, 80, 96, 128, 136, 192, 256])
def test_decode_head_dimensions(dim, dtype):
    from moba_opt import PagedKVCache
    from functools import partial
    rand = partial(globals()["rand"], dtype=dtype)
    cache = PagedKVCache(2, 64, 2, dim, page_size=7, chunk_size=12, dtype=dtype)
    k, v = rand((68, 2, dim), 131), rand((68, 2, dim), 132)
    cache.append(k, v, sequence_ids=[0, 1], cu_seqlens=[0, 27, 68])
    assert_payload(cache, 0, k[:27], v[:27])
    assert_payload(cache, 1, k[27:], v[27:])
    q = rand((3, 4, dim), 133)
    for mode in ("moba", "dense"):
        check(cache, cache.attend(q, sequence_ids=[0, 1, 1], positions=[26, 40, 5], topk=2, mode=mode), q)


@pytest.mark.parametrize("page", [1, 3, 7, 16, 31, 48, 64])
def test_pages_and_chunks_need_not_align(page):
    from moba_opt import PagedKVCache
    cache = PagedKVCache(1, 97, 2, 80, page_size=page, chunk_size=24)
    cache.k_cache.fill_(float("nan"))
    cache.v_cache.fill_(float("nan"))
    k, v = rand((79, 2, 80), 141), rand((79, 2, 80), 142)
    cache.append(k, v, sequence_ids=[0], cu_seqlens=[0, 79])
    assert_payload(cache, 0, k, v)
    q = rand((2, 8, 80), 143)
    for topk in (1, 2, 9):
        check(cache, cache.attend(q, sequence_ids=[0, 0], positions=[0, 78], topk=topk), q)


def test_recycled_pages_and_request_isolation():
    from moba_opt import PagedKVCache
    cache = PagedKVCache(3, 12, 1, 16, page_size=3, num_pages=4, chunk_size=4)
    cache.append(rand((9, 1, 16), 151), rand((9, 1, 16), 152), sequence_ids=[0, 1], cu_seqlens=[0, 6, 9])
    q = rand((1, 4, 16), 153)
    before = cache.attend(q, sequence_ids=[1], mode="dense").output.clone()
    cache.reset([0])
    cache.append(rand((6, 1, 16), 154), rand((6, 1, 16), 155), sequence_ids=[2], cu_seqlens=[0, 6])
    assert cache.page_table[2][:2] == (1, 0)
    assert torch.equal(cache.attend(q, sequence_ids=[1], mode="dense").output, before)
    check(cache, cache.attend(q, sequence_ids=[2], topk=2), q)
    with pytest.raises(ValueError, match="cached tokens"):
        cache.attend(q, sequence_ids=[0])


def test_chunked_append_is_causal():
    from moba_opt import PagedKVCache
    k, v = rand((19, 2, 32), 161), rand((19, 2, 32), 162)
    q = rand((7, 8, 32), 163)
    cache = PagedKVCache(2, 32, 2, 32, page_size=3, chunk_size=4)
    cache.append(torch.cat((k[:5], k[9:16])), torch.cat((v[:5], v[9:16])), sequence_ids=[0, 1], cu_seqlens=[0, 5, 12])
    result = cache.append_and_attend(q, torch.cat((k[5:9], k[16:])), torch.cat((v[5:9], v[16:])), sequence_ids=[0, 1],
                                     cu_seqlens=[0, 4, 7], topk=2)
    assert_payload(cache, 0, k[:9], v[:9])
    assert_payload(cache, 1, k[9:], v[9:])
    assert result.positions == (5, 6, 7, 8, 7, 8, 9)
    check(cache, result, q)
    other = PagedKVCache(2, 32, 2, 32, page_size=3, chunk_size=4)
    k2, v2 = k.clone(), v.clone()
    k2[6:9] = 100
    v2[6:9] = -100
    other.append(k2, v2, sequence_ids=[0, 1], cu_seqlens=[0, 9, 19])
    compare = other.attend(q[:1], sequence_ids=[0], positions=[5], topk=2)
    torch.testing.assert_close(compare.output, result.output[:1], atol=0.02, rtol=0.02)


def test_routing_is_per_query_head_and_uses_only_closed_history():
    from moba_opt import PagedKVCache
    cache = PagedKVCache(1, 16, 2, 8, page_size=3, chunk_size=4)
    k = torch.zeros(13, 2, 8, device="cuda", dtype=cache.dtype)
    for block in range(4):
        k[block * 4:min((block + 1) * 4, 13), 0, 0] = block + 1
        k[block * 4:min((block + 1) * 4, 13), 1, 0] = 4 - block
    cache.append(k, rand(k.shape, 171), sequence_ids=[0], cu_seqlens=[0, 13])
    q = torch.zeros(2, 4, 8, device="cuda", dtype=cache.dtype)
    q[:, :, 0] = 1
    result = cache.attend(q, sequence_ids=[0, 0], positions=[12, 7], topk=3)
    route = result.selected_blocks.cpu()
    assert route[0, 0].tolist() == [3, 2, 1]       # descending score order after the own chunk
    assert route[0, 2].tolist() == [3, 0, 1]
    assert route[1, 0].tolist() == [1, 0, -1]
    check(cache, result, q)


def test_exact_ties_choose_the_lowest_chunk():
    from moba_opt import PagedKVCache
    cache = PagedKVCache(1, 64, 1, 8, page_size=4, chunk_size=4)
    k = torch.ones(33, 1, 8, device="cuda", dtype=cache.dtype)      # every chunk mean identical
    cache.append(k, rand(k.shape, 172), sequence_ids=[0], cu_seqlens=[0, 33])
    q = torch.ones(1, 2, 8, device="cuda", dtype=cache.dtype)
    result = cache.attend(q, sequence_ids=[0], topk=4)
    assert result.selected_blocks[0, 0].tolist() == [8, 0, 1, 2]
    assert result.selected_blocks[0, 1].tolist() == [8, 0, 1, 2]


def test_append_partition_invariance():
    from moba_opt import PagedKVCache
    k, v = rand((25, 2, 24), 181), rand((25, 2, 24), 182)
    a = PagedKVCache(1, 32, 2, 24, page_size=7, chunk_size=6)
    b = PagedKVCache(1, 32, 2, 24, page_size=7, chunk_size=6)
    a.append(k, v, sequence_ids=[0], cu_seqlens=[0, 25])
    for lo, hi in [(0, 1), (1, 5), (5, 13), (13, 25)]:
        b.append(k[lo:hi], v[lo:hi], sequence_ids=[0], cu_seqlens=[0, hi - lo])
    assert torch.equal(a._means[:, :4], b._means[:, :4])
    q = rand((1, 8, 24), 183)
    x, y = a.attend(q, sequence_ids=[0], topk=3), b.attend(q, sequence_ids=[0], topk=3)
    assert torch.equal(x.output, y.output)


@pytest.mark.parametrize("hq,hk", [(8, 1), (8, 2), (28, 4)])
def test_decode_matches_last_prefill_row(hq, hk):
    from moba_opt import PagedKVCache
    from moba_opt.api import run_impl
    q, k, v = rand((97, hq, 64), 191), rand((97, hk, 64), 192), rand((97, hk, 64), 193)
    cu = torch.tensor([0, 97], device="cuda", dtype=torch.int32)
    ref = run_impl("opt_gqa_cuda", q, k, v, cu, 97, {"chunk_size": 16, "topk": 3})[-1:]
    cache = PagedKVCache(1, 128, hk, 64, page_size=7, chunk_size=16)
    cache.append(k, v, sequence_ids=[0], cu_seqlens=[0, 97])
    result = cache.attend(q[-1:], sequence_ids=[0], topk=3)
    torch.testing.assert_close(result.output, ref, atol=0.02, rtol=0.02)
    check(cache, result, q[-1:])


def test_errors_do_not_mutate_cache():
    from moba_opt import PagedKVCache
    cache = PagedKVCache(2, 8, 1, 16, page_size=3, num_pages=1, chunk_size=4)
    q = rand((1, 4, 16), 201)
    with pytest.raises(ValueError, match="cached tokens"):
        cache.attend(q, sequence_ids=[0])
    k, v = rand((3, 1, 16), 202), rand((3, 1, 16), 203)
    cache.append(k, v, sequence_ids=[0], cu_seqlens=[0, 3])
    before = cache.materialize(0)
    with pytest.raises(ValueError, match="pool exhausted"):
        cache.append(k[:1], v[:1], sequence_ids=[1])
    assert cache.lengths == (3, 0)
    for actual, expected in zip(cache.materialize(0), before):
        assert torch.equal(actual, expected)
    with pytest.raises(ValueError, match="inference-only"):
        cache.append_and_attend(q.clone().requires_grad_(True), k[:1], v[:1], sequence_ids=[0])
    with pytest.raises(ValueError, match="NaN/Inf"):
        cache.append(torch.full_like(k[:1], float("nan")), v[:1], sequence_ids=[1])
    assert cache.lengths == (3, 0)


def test_cross_stream_is_rejected():
    from moba_opt import PagedKVCache
    cache = PagedKVCache(1, 8, 1, 8, page_size=3, chunk_size=4)
    k, v = rand((3, 1, 8), 211), rand((3, 1, 8), 212)
    cache.append(k, v, sequence_ids=[0], cu_seqlens=[0, 3])
    q = rand((1, 1, 8), 213)
    with torch.cuda.stream(torch.cuda.Stream()):
        with pytest.raises(ValueError, match="cross-stream"):
            cache.attend(q, sequence_ids=[0])
    check(cache, cache.attend(q, sequence_ids=[0]), q)


def test_long_context_single_token_decode():
    from moba_opt import PagedKVCache
    cache = PagedKVCache(1, 8193, 8, 128, page_size=16, chunk_size=128)
    cache.append(rand((8192, 8, 128), 221), rand((8192, 8, 128), 222), sequence_ids=[0], cu_seqlens=[0, 8192])
    q, k, v = rand((1, 32, 128), 223), rand((1, 8, 128), 224), rand((1, 8, 128), 225)
    result = cache.append_and_attend(q, k, v, sequence_ids=[0], topk=4)
    assert cache.lengths == (8193,) and result.positions == (8192,)
    check(cache, result, q)


@pytest.mark.parametrize("chunk,dim,length,page", [(1, 8, 5, 3), (1024, 256, 1025, 3), (2048, 128, 4500, 48)])
def test_chunk_size_extremes(chunk, dim, length, page):
    from moba_opt import PagedKVCache
    cache = PagedKVCache(1, length + 1, 1, dim, page_size=page, chunk_size=chunk)
    cache.append(rand((length, 1, dim), 231), rand((length, 1, dim), 232), sequence_ids=[0], cu_seqlens=[0, length])
    q = rand((1, 4, dim), 233)
    check(cache, cache.attend(q, sequence_ids=[0], topk=2), q)
    check(cache, cache.attend(q, sequence_ids=[0], mode="dense"), q)


@pytest.mark.parametrize("hq,dim,chunk,length,kernel", [
    (32, 32, 4, 700, CLUSTER_16), (8, 64, 1, 1100, CLUSTER_16), (7, 64, 2, 300, CLUSTER_16),   # merged without partials in memory
    (32, 32, 64, 12790, FIXED),          # weights of 64 of 200 partials fit, and no sums
    (16, 64, 64, 19190, FIXED),          # 256 of 300
    (32, 32, 128, 12790, FIXED_DEEP),    # the weights of all 100 partials, the sums of 9
    (32, 32, 64, 66500, STREAMED),       # 260 shares of the one pair, weights of 256 would fit
])
def test_dense_merge_over_more_partials_than_fit_in_shared_memory(hq, dim, chunk, length, kernel):
    """The merge keeps weights and sums of a head's partials in shared memory up to a capacity that shrinks with the group
    size; the partials beyond it are read and weighted from memory.  A cluster keeps none."""
    from moba_opt import PagedKVCache
    cache = PagedKVCache(1, length + 1, 1, dim, page_size=16, chunk_size=chunk)
    cache.append(rand((length, 1, dim), 271), rand((length, 1, dim), 272), sequence_ids=[0], cu_seqlens=[0, length])
    taken = attend_kernels(cache)
    q = rand((1, hq, dim), 273)
    check(cache, cache.attend(q, sequence_ids=[0], mode="dense"), q)
    assert taken == [kernel]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("dim", [32, 64, 128, 256])
@pytest.mark.parametrize("mode,chunk,topk,kernel", [
    ("dense", 2048, 4, FIXED_DEEP),      # 12 pairs x 6 chunks x 2 parts of 1024 tokens: a ring wraps in each team
    ("moba", 2048, 3, FIXED_DEEP),
    ("dense", 512, 4, FIXED),            # 288 CTAs
    ("moba", 512, 9, FIXED),
])
def test_fixed_parts(mode, chunk, topk, kernel, dim, dtype):
    """A CTA per part of a chunk, whole parts and ragged last ones, with one team of warps and with two (above head dimension
    128 always one, and a dense grid of more than one CTA per SM is streamed)."""
    from moba_opt import PagedKVCache
    lens = [12000, 5003, 70]
    cache = PagedKVCache(3, 12288, 4, dim, page_size=48, chunk_size=chunk, dtype=dtype)
    cu = np.concatenate(([0], np.cumsum(lens))).tolist()
    k, v = rand((cu[-1], 4, dim), 275, dtype), rand((cu[-1], 4, dim), 276, dtype)
    cache.append_prefill(k, v, sequence_ids=[0, 1, 2], cu_seqlens=cu)
    taken = attend_kernels(cache)
    q = rand((3, 8, dim), 277, dtype)
    result = cache.attend(q, sequence_ids=[0, 1, 2], topk=topk, mode=mode)
    check(cache, result, q)
    again = cache.attend(q, sequence_ids=[0, 1, 2], topk=topk, mode=mode)
    assert torch.equal(result.output, again.output) and torch.equal(result.lse, again.lse)
    assert taken == [STREAMED if (dim, mode, kernel) == (256, "dense", FIXED) else kernel] * 2


@pytest.mark.parametrize("page,chunk,dim,hk", [(16, 32, 64, 2), (7, 24, 40, 3), (48, 128, 128, 1), (3, 1, 8, 2), (16, 512, 64, 2)])
def test_prefill_hand_off_equals_append(page, chunk, dim, hk):
    """`append_prefill` (one launch: pages + means in one pass over K) leaves the cache exactly as `append` does:
    payload, lengths, page table and chunk means bit for bit, for ragged prompts, prompts that continue a sequence in
    the middle of a chunk, and prompts shorter than a chunk."""
    from moba_opt import PagedKVCache
    first = [chunk + 5, 3, 2 * chunk]
    second = [max(2, 3 * chunk - 7), chunk // 2 + 1, 1]
    caches = [PagedKVCache(3, sum(map(max, zip(first, second))) * 2 + 4 * chunk, hk, dim, page_size=page, chunk_size=chunk)
              for _ in range(2)]
    for round_, counts in enumerate((first, second)):
        total = sum(counts)
        k, v = rand((total, hk, dim), 281 + round_), rand((total, hk, dim), 291 + round_)
        cu = [0]
        for n in counts:
            cu.append(cu[-1] + n)
        order = [2, 0, 1] if round_ else [0, 1, 2]
        caches[0].append(k, v, sequence_ids=order, cu_seqlens=cu)
        lengths = caches[1].append_prefill(k, v, sequence_ids=order, cu_seqlens=cu)
        assert caches[0].lengths == caches[1].lengths and caches[0].page_table == caches[1].page_table
        assert lengths == tuple(caches[1].lengths[s] for s in order)
        for sid in range(3):
            a, b = caches[0].materialize(sid), caches[1].materialize(sid)
            assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
            closed = caches[0].lengths[sid] // chunk
            assert torch.equal(caches[0]._means[sid, :closed], caches[1]._means[sid, :closed])
    q = rand((3, 2 * hk, dim), 299)
    check(caches[1], caches[1].attend(q, sequence_ids=[0, 1, 2], topk=3), q)


def test_prefill_hand_off_errors_do_not_mutate_cache():
    from moba_opt import PagedKVCache
    cache = PagedKVCache(1, 64, 1, 8, page_size=4, chunk_size=8)
    k = rand((10, 1, 8), 301)
    cache.append_prefill(k, k.clone(), sequence_ids=[0], cu_seqlens=[0, 10])
    lengths, table = cache.lengths, cache.page_table
    with pytest.raises(ValueError):
        cache.append_prefill(rand((60, 1, 8), 302), rand((60, 1, 8), 303), sequence_ids=[0], cu_seqlens=[0, 60])   # over capacity
    with pytest.raises(ValueError):
        cache.append_prefill(k, k.clone(), sequence_ids=[0], cu_seqlens=[0, 9])                                    # bad cu_seqlens
    assert cache.lengths == lengths and cache.page_table == table
    got = cache.materialize(0)
    assert torch.equal(got[0], k)


def test_extreme_logits_use_stable_online_softmax():
    from moba_opt import PagedKVCache
    cache = PagedKVCache(1, 16, 1, 8, page_size=3, chunk_size=4)
    k = torch.full((13, 1, 8), 1000.0, device="cuda", dtype=cache.dtype)
    k[::2] = -1000
    cache.append(k, rand((13, 1, 8), 241), sequence_ids=[0], cu_seqlens=[0, 13])
    q = torch.full((1, 2, 8), 1000.0, device="cuda", dtype=cache.dtype)
    q[:, 1] = -1000
    check(cache, cache.attend(q, sequence_ids=[0], mode="dense"), q)


def test_maximum_topk_with_nonstandard_heads_and_ragged_queries():
    from moba_opt import PagedKVCache
    cache = PagedKVCache(3, 97, 3, 40, page_size=7, chunk_size=8)
    cache.append(rand((153, 3, 40), 261), rand((153, 3, 40), 262), sequence_ids=[0, 1, 2], cu_seqlens=[0, 81, 88, 153])
    q = rand((4, 15, 40), 263)
    result = cache.attend(q, sequence_ids=[2, 0, 1, 2], positions=[64, 80, 6, 23], topk=9)
    assert result.selected_blocks.shape == (4, 15, 9)
    assert (result.selected_blocks[2, :, 1:] == -1).all()
    check(cache, result, q)


@pytest.mark.parametrize("combined", [False, True])
def test_append_rejects_aliases_before_mutation(combined):
    from moba_opt import PagedKVCache
    cache = PagedKVCache(1, 8, 1, 8, page_size=3, chunk_size=4)
    cache.k_cache.zero_()
    cache.v_cache.zero_()
    alias = cache.k_cache.reshape(-1, 1, 8)[:1]
    external = rand((1, 1, 8), 271)
    with pytest.raises(ValueError, match="must not alias"):
        if combined:
            cache.append_and_attend(alias, external, external, sequence_ids=[0])
        else:
            cache.append(alias, external, sequence_ids=[0])
    assert cache.lengths == (0,)
    cache.append(external, external, sequence_ids=[0])
    assert cache.lengths == (1,)


@pytest.mark.parametrize("kwargs", [{"head_dim": 0}, {"head_dim": 264}, {"head_dim": 33}, {"num_kv_heads": 0}, {"page_size": 0},
                                    {"num_pages": 0}, {"chunk_size": 8193}, {"dtype": torch.float32}, {"dtype": torch.float64},
                                    {"device": "cpu"}])
def test_cache_contract_violations(kwargs):
    from moba_opt import PagedKVCache
    cfg = dict(batch_size=1, max_seq_len=16, num_kv_heads=2, head_dim=64)
    cfg.update(kwargs)
    with pytest.raises(ValueError):
        PagedKVCache(**cfg)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("layout", ["whole", "fused", "odd"])
def test_one_finite_check_for_all_inputs(dtype, layout):
    """First and last element of each tensor, NaN and both infinities; the largest finite values pass.  `fused`: views of
    one projection's output (16-byte aligned rows); `odd`: rows that start on 2-byte boundaries, read element by element."""
    from moba_opt import PagedKVCache
    tokens, hq, hk, d = 37, 6, 2, 24
    cache = PagedKVCache(1, 64, hk, d, dtype=dtype)
    if layout == "whole":
        q, k, v = (torch.full((tokens, h, d), torch.finfo(dtype).max, device="cuda", dtype=dtype) for h in (hq, hk, hk))
    else:
        pad = 0 if layout == "fused" else 1
        qkv = torch.full((tokens, hq + 2 * hk, d + pad), torch.finfo(dtype).min, device="cuda", dtype=dtype)[..., pad:]
        q, k, v = qkv[:, :hq], qkv[:, hq:hq + hk], qkv[:, hq + hk:]
    named = [("k", k), ("v", v), ("q", q)]
    cache._finite.require(named)
    for name, t in named:
        for at in ((0, 0, 0), (tokens - 1, t.shape[1] - 1, d - 1), (tokens // 2, 0, 11)):
            for bad in (float("nan"), float("inf"), float("-inf")):
                keep = t[at].clone()
                t[at] = bad
                with pytest.raises(ValueError, match=f"{name} contains NaN/Inf"):
                    cache._finite.require(named)
                t[at] = keep
    cache._finite.require(named)


def test_the_first_input_at_fault_is_reported():
    """One finite check covers all inputs of a call, but a tensor's NaN comes before the faults of the tensors after it, and a
    fault of shape before the NaN of a later one; nothing reaches the cache or the plan's positions."""
    from moba_opt import PagedKVCache
    cache = PagedKVCache(1, 64, 2, 16)
    k, v, q = rand((3, 2, 16), 341), rand((3, 2, 16), 342), rand((3, 4, 16), 343)
    cache.append(k, v, sequence_ids=[0], cu_seqlens=[0, 3])
    before = [t.clone() for t in cache.materialize(0)]
    nan = float("nan")
    bad_k, bad_v, bad_q = torch.full_like(k, nan), torch.full_like(v, nan), torch.full_like(q, nan)
    faults = [
        (dict(q=q, k=bad_k, v=v[:, :1]), "k contains NaN/Inf"),
        (dict(q=q, k=k[:, :1], v=bad_v), "k KV head count differs"),
        (dict(q=q[:2], k=k, v=bad_v), "v contains NaN/Inf"),
        (dict(q=bad_q, k=k, v=v[:2]), "v token count differs"),
        (dict(q=bad_q, k=bad_k, v=bad_v), "k contains NaN/Inf"),
        (dict(q=bad_q, k=k, v=v), "q contains NaN/Inf"),
        (dict(q=q[:, :3], k=k, v=v), "multiple of Hkv"),
    ]
    for tensors, message in faults:
        with pytest.raises(ValueError, match=message):
            cache.append_and_attend(**tensors, sequence_ids=[0], cu_seqlens=[0, 3])
    with pytest.raises(ValueError, match="k contains NaN/Inf"):
        cache.append(bad_k, v[:, :1], sequence_ids=[0], cu_seqlens=[0, 3])
    plan = cache.prepare_decode([0], 4, check_finite=True)
    step = [t[:1].contiguous() for t in (q, k, v, bad_q, bad_k)]
    for tensors, message in [((step[3], step[1][:, :1], step[2]), "q contains NaN/Inf"), ((step[0][:, :3], step[4], step[2]), "q must have fixed shape"),
                             ((step[0], step[4], step[2][:, :1]), "k contains NaN/Inf")]:
        with pytest.raises(ValueError, match=message):
            plan.step(*tensors)
    plan.close()
    assert cache.lengths == (3,)
    for got, want in zip(cache.materialize(0), before):
        assert torch.equal(got, want)


@pytest.mark.parametrize("repeat", [1, 8])      # 22 queries: fixed parts, but for three of the dense grids; 176: streamed
@pytest.mark.parametrize("mode", ["moba", "dense"])
@pytest.mark.parametrize("hq,hkv,dim,chunk,page,dtype", [
    (4, 2, 64, 100, 7, torch.bfloat16),      # the last stage of a chunk is part of one
    (6, 1, 32, 64, 16, torch.float16),       # a stage is a chunk
    (40, 2, 96, 130, 48, torch.bfloat16),    # two head blocks per pair, padded head dimension
    (5, 5, 128, 192, 16, torch.float16),
    (2, 1, 256, 70, 3, torch.bfloat16),      # one CTA per SM
])
def test_attend_divides_uneven_work(repeat, mode, hq, hkv, dim, chunk, page, dtype):
    """Fixed parts, or, streamed, equal shares of one list of stages: contexts from one token to many chunks, shares that
    begin and end inside a chunk, several requests in a share and several shares in a request, repeatable bits."""
    from moba_opt import PagedKVCache
    lens = [1, 63, 64, 65, 900, 2, chunk, chunk + 1, 700, 1, 333, 1024, 5, 640, 129, 77, 2 * chunk, 511]
    cache = PagedKVCache(len(lens), 1024, hkv, dim, page_size=page, chunk_size=chunk, dtype=dtype)
    cu = np.concatenate(([0], np.cumsum(lens))).tolist()
    k, v = rand((cu[-1], hkv, dim), 71, dtype), rand((cu[-1], hkv, dim), 72, dtype)
    cache.append_prefill(k, v, sequence_ids=list(range(len(lens))), cu_seqlens=cu)
    ids = (list(range(len(lens))) + [4, 11, 11, 8]) * repeat           # several queries of a request, some not at its end
    positions = ([n - 1 for n in lens] + [450, 1000, 63, 0]) * repeat
    q = rand((len(ids), hq, dim), 73, dtype)
    taken = attend_kernels(cache)
    result = cache.attend(q, sequence_ids=ids, positions=positions, topk=4, mode=mode)
    check(cache, result, q)
    again = cache.attend(q, sequence_ids=ids, positions=positions, topk=4, mode=mode)
    assert torch.equal(result.output, again.output) and torch.equal(result.lse, again.lse)
    assert taken == [FIXED if repeat == 1 and (mode == "moba" or dim in (32, 96)) else STREAMED] * 2


@pytest.mark.parametrize("mode", ["moba", "dense"])
@pytest.mark.parametrize("lens,hq,hkv,dim,chunk,page,dtype", [
    ((1,), 4, 1, 64, 100, 7, torch.bfloat16),             # fewer stages than CTAs in the cluster
    ((1000,), 14, 2, 64, 100, 16, torch.bfloat16),        # the last stage of a chunk is part of one
    ((63, 64, 65), 32, 1, 32, 64, 16, torch.float16),     # two head blocks, a stage is a chunk
    ((640, 5, 129), 6, 2, 96, 130, 48, torch.bfloat16),   # six pairs: clusters of eight
    ((511, 700), 4, 4, 128, 192, 16, torch.float16),
    ((900, 71), 2, 1, 256, 70, 3, torch.bfloat16),        # one team per CTA
])
def test_cluster_attend_divides_a_request(lens, mode, hq, hkv, dim, chunk, page, dtype):
    """Small batches: the stages of a (request, kv head) pair over the CTAs of a cluster, repeatable bits."""
    from moba_opt import PagedKVCache
    cache = PagedKVCache(len(lens), max(lens) + 8, hkv, dim, page_size=page, chunk_size=chunk, dtype=dtype)
    cu = np.concatenate(([0], np.cumsum(lens))).tolist()
    k, v = rand((cu[-1], hkv, dim), 81, dtype), rand((cu[-1], hkv, dim), 82, dtype)
    cache.append_prefill(k, v, sequence_ids=list(range(len(lens))), cu_seqlens=cu)
    q = rand((len(lens), hq, dim), 83, dtype)
    taken = attend_kernels(cache)
    result = cache.attend(q, sequence_ids=list(range(len(lens))), topk=4, mode=mode)
    check(cache, result, q)
    again = cache.attend(q, sequence_ids=list(range(len(lens))), topk=4, mode=mode)
    assert torch.equal(result.output, again.output) and torch.equal(result.lse, again.lse)
    assert taken == [CLUSTER_16 if len(lens) * hkv <= 4 else CLUSTER_8] * 2


@pytest.mark.parametrize("mode,chunk", [("dense", 512), ("moba", 512), ("moba", 100)])
@pytest.mark.parametrize("rows,kernel", [(1, CLUSTER_16), (160, STREAMED)])
def test_lookups_step_over_pages_of_any_size(rows, kernel, mode, chunk):
    """From a stage of 64 tokens to the next the page is stepped, not divided for: any page size gives the same bits."""
    from moba_opt import PagedKVCache
    length = 3001
    k, v, q = rand((length, 2, 64), 361), rand((length, 2, 64), 362), rand((rows, 32, 64), 363)
    first = None
    for page in (1, 3, 48, 63, 64, 65, 200, 4096):
        cache = PagedKVCache(1, 4096, 2, 64, page_size=page, chunk_size=chunk)
        cache.append_prefill(k, v, sequence_ids=[0], cu_seqlens=[0, length])
        taken = attend_kernels(cache)
        result = cache.attend(q, sequence_ids=[0] * rows, positions=[length - 1 - 7 * i for i in range(rows)], topk=4, mode=mode)
        assert taken == [kernel]
        if first is None:
            first = result
            check(cache, result, q)
        assert torch.equal(first.output, result.output) and torch.equal(first.lse, result.lse)


@pytest.mark.parametrize("requests,length", [(200, 40), (64, 300), (64, 330), (30, 700)])
def test_streamed_shares_of_short_requests(requests, length):
    """Requests of a few stages in a cache for many more: a share is an eighth of an average pair, down to one stage."""
    from moba_opt import PagedKVCache
    cache = PagedKVCache(requests, 16384, 2, 64, page_size=16, num_pages=requests * 64, chunk_size=512)
    lens = [length - i % 7 for i in range(requests)]
    cu = np.concatenate(([0], np.cumsum(lens))).tolist()
    cache.append_prefill(rand((cu[-1], 2, 64), 371), rand((cu[-1], 2, 64), 372), sequence_ids=list(range(requests)), cu_seqlens=cu)
    taken = attend_kernels(cache)
    q = rand((requests, 14, 64), 373)
    result = cache.attend(q, sequence_ids=list(range(requests)), mode="dense")
    check(cache, result, q)
    again = cache.attend(q, sequence_ids=list(range(requests)), mode="dense")
    assert torch.equal(result.output, again.output) and taken == [STREAMED] * 2


@pytest.mark.parametrize("layout", ["fused", "heads_first", "expanded", "unaligned"])
def test_append_reads_strided_views(layout):
    """Views of a fused projection, a transposed layout, one head for all and rows off the 16-byte grid give the cache that
    contiguous tensors give: pages and chunk means bit for bit."""
    from moba_opt import PagedKVCache
    tokens, hkv, dim = 300, 2, 40
    if layout == "fused":
        qkv = rand((tokens, 3 * hkv, dim), 91)
        k, v = qkv[:, hkv:2 * hkv], qkv[:, 2 * hkv:]
    elif layout == "heads_first":
        k, v = (rand((hkv, tokens, dim), s).transpose(0, 1) for s in (92, 93))
    elif layout == "expanded":
        k, v = (rand((tokens, 1, dim), s).expand(tokens, hkv, dim) for s in (94, 95))
    else:
        k, v = (rand((tokens * hkv * dim + 1,), s)[1:].view(tokens, hkv, dim) for s in (96, 97))
    caches = [PagedKVCache(2, 512, hkv, dim, page_size=7, chunk_size=64) for _ in range(2)]
    for cache, (kk, vv) in zip(caches, ((k, v), (k.clone(memory_format=torch.contiguous_format), v.clone(memory_format=torch.contiguous_format)))):
        cache.append(kk, vv, sequence_ids=[0, 1], cu_seqlens=[0, 130, tokens])
    for sid in range(2):
        assert_payload(caches[0], sid, *caches[1].materialize(sid))
        closed = caches[0].lengths[sid] // 64
        assert torch.equal(caches[0]._means[sid, :closed], caches[1]._means[sid, :closed])
    assert_payload(caches[0], 0, k[:130], v[:130])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("requests,queries,hq,hkv,dim,length,mode", [
    (12, 1, 16, 4, 128, 6100, "dense"),      # streamed: 576 parts of 512 tokens do not fit the GPU at once
    (12, 3, 16, 4, 64, 6100, "moba"),        # streamed: 36 rows x 4 heads, up to 12 of 12 chunks in a union
    (1, 1, 14, 2, 64, 6100, "dense"),        # a cluster per pair
    (2, 1, 8, 4, 128, 2900, "dense"),
    (1, 2, 14, 2, 64, 6100, "moba"),
])
def test_probabilities_keep_more_than_16_bits(requests, queries, hq, hkv, dim, length, mode, dtype):
    """Where a warp's run of tokens is longer than a fixed part, P is multiplied in two 16-bit pieces.  Each p is then off by at
    most 2^-16 (2^-22) of itself and the sums by FP32 rounding, against 2^-9 (2^-12) for the rounding of the output: what
    is left is the error of the oracle's own result rounded once, within 2 % (5 % in half precision, where the FP32
    parts - scores of magnitude up to 6 off by 2^-21, exp2 by 2^-22 - are closer to it).  With P rounded once it is 20 to 30 % more."""
    from moba_opt import PagedKVCache
    cache = PagedKVCache(requests, length, hkv, dim, page_size=48, chunk_size=512, dtype=dtype)
    lens = [length - 37 * i for i in range(requests)]
    cu = np.concatenate(([0], np.cumsum(lens))).tolist()
    k, v = rand((cu[-1], hkv, dim), 301, dtype), rand((cu[-1], hkv, dim), 302, dtype)
    cache.append_prefill(k, v, sequence_ids=list(range(requests)), cu_seqlens=cu)
    ids = [i for i in range(requests) for _ in range(queries)]
    positions = [lens[i] - 1 - 500 * j for i in range(requests) for j in range(queries)]
    q = rand((len(ids), hq, dim), 303, dtype)
    taken = attend_kernels(cache)
    result = cache.attend(q, sequence_ids=ids, positions=positions, topk=4, mode=mode)
    check(cache, result, q)
    assert taken[0] in ((STREAMED,) if requests == 12 else (CLUSTER_8, CLUSTER_16))
    keys, values = zip(*[[torch_to_f64(t) for t in cache.materialize(i)] for i in range(requests)])
    sel = None if result.selected_blocks is None else result.selected_blocks.cpu().numpy()
    want, _ = mo.decode_attend(torch_to_f64(q), keys, values, ids, positions, 512, sel)
    rounded = torch_to_f64(torch.from_numpy(want).to(dtype))
    error, least = np.linalg.norm(torch_to_f64(result.output) - want), np.linalg.norm(rounded - want)
    assert error <= (1.02 if dtype == torch.bfloat16 else 1.05) * least, f"{error / least:.4f}"


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("rows,hq,hkv,dim,dtype,kernel", [
    (1, 8, 2, 64, torch.bfloat16, CLUSTER_16),
    (2, 6, 1, 128, torch.float16, CLUSTER_16),
    (20, 8, 2, 64, torch.bfloat16, FIXED),
    (4, 40, 2, 128, torch.bfloat16, CLUSTER_8),      # two head blocks
    (20, 40, 2, 128, torch.bfloat16, FIXED),
    (120, 8, 2, 64, torch.float16, STREAMED),
    (80, 40, 2, 96, torch.bfloat16, STREAMED),       # two head blocks
])
def test_values_of_a_chunk_reach_only_the_heads_that_selected_it(rows, hq, hkv, dim, dtype, kernel, bad):
    """A V that is not finite (a caller may switch the check off) spoils the heads that attend its chunk; the others keep
    their bits, whichever kernel runs."""
    from moba_opt import PagedKVCache
    chunk, chunks, poisoned = 100, 6, 2
    length = chunks * chunk + 41
    k, v = rand((length, hkv, dim), 311, dtype), rand((length, hkv, dim), 312, dtype)
    k[:, :, :chunks] = 0
    for c in range(chunks):
        k[c * chunk:(c + 1) * chunk, :, c] = 8                     # chunk c is the best match of a query along axis c
    q = rand((rows, hq, dim), 313, dtype)
    for h in range(hq):
        q[:, h, h % chunks] = 40
    caches = []
    for value in (1.0, bad):
        vv = v.clone()
        vv[poisoned * chunk + 33, :, 5] = value
        vv[poisoned * chunk + 99, :, dim - 1] = value
        cache = PagedKVCache(2, length, hkv, dim, page_size=7, chunk_size=chunk, dtype=dtype)
        cache.check_finite = False
        cache.append(torch.cat((k, k)), torch.cat((vv, vv)), sequence_ids=[0, 1], cu_seqlens=[0, length, 2 * length])
        taken = attend_kernels(cache)
        caches.append(cache.attend(q, sequence_ids=[i % 2 for i in range(rows)], topk=2))
        assert taken == [kernel]
    good, spoiled = caches
    reads = (good.selected_blocks == poisoned).any(-1)
    assert torch.equal(good.selected_blocks, spoiled.selected_blocks) and reads.any() and not reads.all()
    assert torch.equal(good.output[~reads], spoiled.output[~reads]) and torch.equal(good.lse, spoiled.lse)
    assert not spoiled.output[reads][:, 5].isfinite().any() and bool(good.output.isfinite().all())
    if bad == bad:                                                 # an infinity stays one, of its sign
        assert (spoiled.output[reads][:, 5] == bad).all()


def test_threads_with_groups_of_different_size():
    """The cluster kernel's shared memory grows with the group; the limit that a launch sets belongs to the function, so a
    cache with small groups in one thread must not lower it under a launch of another."""
    import ctypes
    from moba_opt import PagedKVCache
    calls, keep = [], []
    for group in (32, 9):
        cache = PagedKVCache(1, 512, 1, 128, chunk_size=64)
        cache.append(rand((300, 1, 128), 321), rand((300, 1, 128), 322), sequence_ids=[0], cu_seqlens=[0, 300])
        p = cache.prepare_decode([0], group, mode="dense", check_finite=False)
        p.launch("attend")
        desc = cache._desc()
        calls.append((p._lib.moba_decode_attend, (
            ctypes.byref(desc), p.q.data_ptr(), p.gpu_ids.data_ptr(), p.positions.data_ptr(), 1, group, None, p._slots, None, None, None, 1,
            p._workspace.data_ptr(), p._ws_bytes, p.output.data_ptr(), p.lse.data_ptr(), cache._status.data_ptr(), p._stream())))
        keep.append((p, desc))
    assert two_threads(calls) == [0, 0]


def test_threads_with_caches_of_different_width():
    """The same for routing, whose shared memory grows with the number of chunks a query may be routed to."""
    import ctypes
    from moba_opt import PagedKVCache
    calls, keep = [], []
    for width in (600, 400):
        cache = PagedKVCache(1, width * 16 + 1, 1, 64, chunk_size=16)
        cache.append(rand((300, 1, 64), 331), rand((300, 1, 64), 332), sequence_ids=[0], cu_seqlens=[0, 300])
        p = cache.prepare_decode([0], 32, check_finite=False)
        assert p.width == width
        p.launch("attend")
        desc = cache._desc()
        calls.append((p._lib.moba_decode_route, (
            ctypes.byref(desc), p.q.data_ptr(), p.gpu_ids.data_ptr(), p.positions.data_ptr(), 1, 32, p.remote, p.width, p.scores.data_ptr(),
            p.selected.data_ptr(), p._u_chunk.data_ptr(), p._u_mask.data_ptr(), p._u_count.data_ptr(), p._stream())))
        keep.append((p, desc))
    assert two_threads(calls) == [0, 0]


def test_the_alias_check_looks_at_the_pools_in_use():
    """Pools that a caller has put in the place of the first ones (offloaded and brought back, say) count, the first ones no longer."""
    from moba_opt import PagedKVCache
    cache = PagedKVCache(1, 8, 1, 8, page_size=3, chunk_size=4)
    first = cache.k_cache.zero_()
    cache.v_cache.zero_()
    cache.k_cache = first.clone()
    external = rand((1, 1, 8), 271)
    with pytest.raises(ValueError, match="must not alias"):
        cache.append(cache.k_cache.reshape(-1, 1, 8)[:1], external, sequence_ids=[0])
    cache.append(first.reshape(-1, 1, 8)[:1], external, sequence_ids=[0])
    assert cache.lengths == (1,)


@pytest.mark.parametrize("counts", [(30, 34), (30, 35), (1, 300)])    # ids and positions as integers, and as arrays
def test_long_segments_in_one_call_equal_append_then_attend(counts):
    from moba_opt import PagedKVCache
    results, n, cu = [], sum(counts), [0, counts[0], sum(counts)]
    first, q, k, v = rand((90, 2, 64), 601), rand((n, 8, 64), 602), rand((n, 2, 64), 603), rand((n, 2, 64), 604)
    for combined in (True, False):
        cache = PagedKVCache(2, 512, 2, 64, page_size=16, chunk_size=32)
        cache.append(first, first, sequence_ids=[1, 0], cu_seqlens=[0, 50, 90])
        if combined:
            results.append(cache.append_and_attend(q, k, v, sequence_ids=[1, 0], cu_seqlens=cu, topk=3))
        else:
            cache.append(k, v, sequence_ids=[1, 0], cu_seqlens=cu)
            ids = [1] * counts[0] + [0] * counts[1]
            results.append(cache.attend(q, sequence_ids=ids, positions=[*range(50, 50 + counts[0]), *range(40, 40 + counts[1])], topk=3))
    a, b = results
    assert a.sequence_ids == b.sequence_ids and a.positions == b.positions and all(type(x) is int for x in a.positions)
    assert torch.equal(a.output, b.output) and torch.equal(a.lse, b.lse) and torch.equal(a.selected_blocks, b.selected_blocks)
