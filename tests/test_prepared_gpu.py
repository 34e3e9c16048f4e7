"""PreparedDecode on the GPU: eager and CUDA-graph steps against the FP64 oracle, capture leaves the
visible cache state untouched, buffer addresses stay fixed, delta uploads happen only on new pages,
and lifecycle / validation errors are atomic (cases of tests/test_prepared_decode.py and
tests/test_decode_routing.py in the reference)."""
import numpy as np
import pytest
import torch

from helpers import torch_to_f64
from oracle import moba_oracle as mo

pytestmark = pytest.mark.gpu


def rand(shape, seed, dtype=torch.bfloat16):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to("cuda", dtype)


def reference(cache, result, q):
    import moba_opt.grouped_attention as ga
    ga.check_status()
    kv = [cache.materialize(i) for i in range(len(cache.lengths))]
    sel = None if result.selected_blocks is None else result.selected_blocks.cpu().numpy()
    out, lse = mo.decode_attend(torch_to_f64(q), [torch_to_f64(x[0]) for x in kv], [torch_to_f64(x[1]) for x in kv],
                                result.sequence_ids, result.positions, cache.chunk_size, sel)
    np.testing.assert_allclose(torch_to_f64(result.output), out, atol=0.02, rtol=0.02)
    np.testing.assert_allclose(torch_to_f64(result.lse), lse, atol=5e-4, rtol=2e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("page,chunk,dim,hq,hk", [(3, 4, 40, 15, 3), (7, 6, 64, 8, 1), (16, 8, 128, 8, 2), (48, 16, 128, 12, 2)])
def test_prepared_steps_match_oracle_and_payload(graph, page, chunk, dim, hq, hk, dtype):
    from moba_opt import PagedKVCache
    from functools import partial
    rand = partial(globals()["rand"], dtype=dtype)
    half = dtype == torch.float16
    cache = PagedKVCache(3, 40, hk, dim, page_size=page, chunk_size=chunk, dtype=dtype)
    k, v = rand((14, hk, dim), 501), rand((14, hk, dim), 502)
    cache.append(k, v, sequence_ids=[2, 0], cu_seqlens=[0, 5, 14])
    stored_k, stored_v = {2: k[:5], 0: k[5:]}, {2: v[:5], 0: v[5:]}
    lengths, table = cache.lengths, cache.page_table
    before = [cache.materialize(s) for s in (2, 0)]
    with cache.prepare_decode([2, 0], hq, topk=3) as plan:
        if graph:
            plan.capture("step").capture("attend")
            assert cache.lengths == lengths and cache.page_table == table
            for sid, (bk, bv) in zip((2, 0), before):
                ak, av = cache.materialize(sid)
                assert torch.equal(ak, bk) and torch.equal(av, bv)
        pointers = [t.data_ptr() for t in (cache._table, cache._lengths, plan.output, plan.scores, plan.selected)]
        for step in range(10):
            q = rand((2, hq, dim), 510 + step)
            kn, vn = rand((2, hk, dim), 530 + step), rand((2, hk, dim), 550 + step)
            result = plan.step(q, kn, vn, use_graph=graph)
            for i, sid in enumerate((2, 0)):
                stored_k[sid] = torch.cat((stored_k[sid], kn[i:i + 1]))
                stored_v[sid] = torch.cat((stored_v[sid], vn[i:i + 1]))
                actual = cache.materialize(sid)
                assert torch.equal(actual[0], stored_k[sid]) and torch.equal(actual[1], stored_v[sid])
            reference(cache, result, q)
            reference(cache, plan.attend(q, use_graph=graph), q)
            closed = cache.lengths[2] // chunk
            if closed:
                want = mo.chunk_means(torch_to_f64(stored_k[2]), chunk, rounding=mo.fp16_round if half else mo.bf16_round)
                np.testing.assert_allclose(torch_to_f64(cache._means[2, :closed]), want, atol=1e-5, rtol=0.002 if half else 0.01)
        assert pointers == [t.data_ptr() for t in (cache._table, cache._lengths, plan.output, plan.scores, plan.selected)]
        assert plan.delta_uploads <= 10
        with pytest.raises(ValueError, match="owns cache"):
            cache.reset()
    cache.reset([2])
    assert cache.lengths == (19, 0, 0)


def test_graph_and_eager_steps_are_bit_identical():
    from moba_opt import PagedKVCache
    outs = []
    for graph in (False, True):
        cache = PagedKVCache(2, 200, 2, 64, page_size=48, chunk_size=16)
        cache.append(rand((150, 2, 64), 701), rand((150, 2, 64), 702), sequence_ids=[0, 1], cu_seqlens=[0, 90, 150])
        with cache.prepare_decode([0, 1], 8, topk=4, check_finite=False) as p:
            if graph:
                p.capture("step")
            seq = []
            for step in range(20):
                r = p.step(rand((2, 8, 64), 710 + step), rand((2, 2, 64), 740 + step), rand((2, 2, 64), 770 + step), use_graph=graph)
                seq.append((r.output.clone(), r.lse.clone(), r.selected_blocks.clone()))
            outs.append(seq)
    for (o1, l1, s1), (o2, l2, s2) in zip(*outs):
        assert torch.equal(o1, o2) and torch.equal(l1, l2) and torch.equal(s1, s2)


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("mode,topk", [("moba", 1), ("dense", 4), ("moba", 9)])
def test_prepared_empty_and_dense_fallback(graph, mode, topk):
    from moba_opt import PagedKVCache
    cache = PagedKVCache(1, 17, 1, 8, page_size=3, chunk_size=4)
    with cache.prepare_decode([0], 4, topk=topk, mode=mode) as p:
        if graph:
            p.capture("step")
        for step in range(9):
            q, kv = rand((1, 4, 8), 601 + step), rand((1, 1, 8), 621 + step)
            reference(cache, p.step(q, kv, kv, use_graph=graph), q)


def test_validation_lifecycle_capacity_and_metadata_delta():
    from moba_opt import PagedKVCache
    c = PagedKVCache(1, 7, 1, 8, page_size=3, chunk_size=4)
    q = torch.ones((1, 1, 8), device="cuda", dtype=c.dtype)
    with c.prepare_decode([0], 1) as p:
        before = c.lengths
        with pytest.raises(ValueError, match="NaN/Inf"):
            p.step(q * float("nan"), q, q)
        with pytest.raises(ValueError, match="capture"):
            p.step(q, q, q, use_graph=True)
        assert c.lengths == before
        for _ in range(7):
            p.step(q, q, q)
        assert p.delta_uploads == 3
        with pytest.raises(ValueError, match="max_seq_len"):
            p.step(q, q, q)
        assert c.lengths == (7,)
        with torch.cuda.stream(torch.cuda.Stream()):
            with pytest.raises(ValueError, match="cross-stream"):
                p.attend(q)
    with pytest.raises(ValueError, match="closed"):
        p.step(q, q, q)
    assert c.lengths == (7,)


def test_input_workspace_alias_and_output_reuse_contract():
    from moba_opt import PagedKVCache
    c = PagedKVCache(1, 8, 1, 8, page_size=3, chunk_size=4)
    q = torch.ones((1, 1, 8), device="cuda", dtype=c.dtype)
    with c.prepare_decode([0], 1, check_finite=False) as p:
        with pytest.raises(ValueError, match="aliases"):
            p.step(p.v, p.k, p.q)
        a = p.step(q, q, q)
        b = p.step(q, q, q)
        assert a.output.data_ptr() == b.output.data_ptr()


def test_capture_after_live_steps_and_graph_capacity_boundary():
    from moba_opt import PagedKVCache
    c = PagedKVCache(1, 4, 1, 8, page_size=1, chunk_size=2)
    q = torch.ones(1, 1, 8, device="cuda", dtype=c.dtype)
    with c.prepare_decode([0], 1) as p:
        for value in (1, 2, 3):
            p.step(q, q, q * value)
        before = c.materialize(0)
        p.capture("step").capture("attend")
        assert c.lengths == (3,)
        assert torch.equal(before[0], c.materialize(0)[0]) and torch.equal(before[1], c.materialize(0)[1])
        reference(c, p.step(q, q, q * 4, use_graph=True), q)
        with pytest.raises(ValueError, match="max_seq_len"):
            p.step(q, q, q, use_graph=True)
        assert c.lengths == (4,)


def test_graph_closes_large_chunk_at_maximum_head_dimension():
    from moba_opt import PagedKVCache
    c = PagedKVCache(1, 2050, 1, 256, page_size=48, chunk_size=2048)
    k, v = rand((2047, 1, 256), 801), rand((2047, 1, 256), 802)
    c.append(k, v, sequence_ids=[0], cu_seqlens=[0, 2047])
    q = rand((1, 4, 256), 803)
    kn, vn = k[:1].clone(), v[:1].clone()
    with c.prepare_decode([0], 4) as p:
        p.capture("step")
        reference(c, p.step(q, kn, vn, use_graph=True), q)
        expected = torch.cat((k, kn)).float().mean(0).to(c.dtype)
        torch.testing.assert_close(c._means[0, 0], expected, atol=1e-5, rtol=0.01)
        reference(c, p.step(q, kn, vn, use_graph=True), q)   # first query that can route to chunk 0


def test_bound_input_buffers_support_graph_without_staging_copies():
    from moba_opt import PagedKVCache
    c = PagedKVCache(1, 8, 1, 8, page_size=4, chunk_size=2)
    with c.prepare_decode([0], 1, check_finite=False) as p:
        p.q.fill_(1)
        p.k.fill_(1)
        p.v.fill_(2)
        p.capture("step")
        for _ in range(3):
            result = p.step(p.q, p.k, p.v, use_graph=True)
            assert torch.equal(result.output, torch.full_like(result.output, 2))
        assert p.delta_uploads == 1
        with pytest.raises(ValueError, match="owns cache"):
            c.prepare_decode([0], 1)


def test_no_history_preserves_padding():
    from moba_opt import PagedKVCache
    cache = PagedKVCache(2, 65, 1, 8, page_size=7, chunk_size=8)
    data = torch.ones(65, 1, 8, device="cuda", dtype=cache.dtype)
    cache.append(data, data, sequence_ids=[1], cu_seqlens=[0, 65])
    q = torch.ones(1, 4, 8, device="cuda", dtype=cache.dtype)
    result = cache.attend(q, sequence_ids=[1], positions=[0], topk=9)
    assert result.selected_blocks.shape == (1, 4, 9)
    assert (result.selected_blocks[:, :, 0] == 0).all()
    assert (result.selected_blocks[:, :, 1:] == -1).all()
    cache.reset()
    assert cache._candidate_count == 0


def test_device_metadata_mirrors_cpu_layout():
    from moba_opt import PagedKVCache
    cache = PagedKVCache(2, 16, 1, 8, page_size=3, chunk_size=4)
    q = torch.ones(3, 4, 8, device="cuda", dtype=cache.dtype)
    kv = torch.ones(3, 1, 8, device="cuda", dtype=cache.dtype)
    result = cache.append_and_attend(q, kv, kv, sequence_ids=[1, 0], cu_seqlens=[0, 2, 3])
    assert result.sequence_ids == (1, 1, 0) and result.positions == (0, 1, 0)
    again = cache.attend(q, sequence_ids=[1, 1, 0], positions=[0, 1, 0])
    assert torch.equal(result.output, again.output)
    assert torch.equal(cache._table.cpu(), torch.tensor(cache.page_table, dtype=torch.int32))
    assert torch.equal(cache._lengths.cpu(), torch.tensor(cache.lengths, dtype=torch.int32))


@pytest.mark.parametrize("bad_name", ["q", "k", "v"])
def test_combined_api_rejects_nonfinite_before_append(bad_name):
    from moba_opt import PagedKVCache
    cache = PagedKVCache(1, 8, 1, 8, page_size=3, chunk_size=4)
    tensors = {"q": torch.ones(1, 4, 8, device="cuda", dtype=cache.dtype), "k": torch.ones(1, 1, 8, device="cuda", dtype=cache.dtype),
               "v": torch.ones(1, 1, 8, device="cuda", dtype=cache.dtype)}
    tensors[bad_name][0, 0, 0] = float("nan")
    with pytest.raises(ValueError, match="NaN/Inf"):
        cache.append_and_attend(**tensors, sequence_ids=[0])
    assert cache.lengths == (0,)


@pytest.mark.parametrize("requests,hq,hk,dim,chunk,page,mode,dtype,start", [
    (1, 14, 2, 64, 32, 16, "moba", torch.bfloat16, 61),     # pages and chunks end together
    (1, 14, 2, 64, 32, 16, "dense", torch.bfloat16, 61),
    (4, 6, 1, 128, 24, 7, "moba", torch.float16, 70),       # a page across a chunk's end
    (2, 40, 2, 96, 16, 1, "moba", torch.bfloat16, 45),      # two head blocks; every token opens a page
    (2, 4, 4, 32, 20, 5, "moba", torch.float16, 18),        # eight CTAs a pair; no candidate at first
    (3, 8, 1, 8, 16, 16, "dense", torch.bfloat16, 1),
])
def test_step_in_one_launch_equals_its_three_launches(requests, hq, hk, dim, chunk, page, mode, dtype, start):
    """A small batch's step is one launch; the entry points it stands for, called one after the other, leave the same routes, scores,
    cache, means and lengths.  The new token's product is exact in one and split in two 16-bit pieces in the other, so outputs may
    round to neighbouring values: one unit in the last place, 2^-7 of the value in bf16 and 2^-10 in half precision."""
    import ctypes
    from moba_opt import PagedKVCache
    gen = torch.Generator().manual_seed(dim + chunk)
    rnd = lambda *shape: torch.randn(*shape, generator=gen).to("cuda", dtype)
    steps = 2 * chunk + 3
    plans, caches = [], []
    lens = [start + 3 * i for i in range(requests)]
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    k0, v0 = rnd(cu[-1], hk, dim), rnd(cu[-1], hk, dim)
    for _ in range(2):
        cache = PagedKVCache(requests, max(lens) + steps, hk, dim, page_size=page, chunk_size=chunk, dtype=dtype)
        cache.append(k0, v0, sequence_ids=list(range(requests)), cu_seqlens=cu)
        caches.append(cache)
        plans.append(cache.prepare_decode(list(range(requests)), hq, topk=3, mode=mode, check_finite=False))
    one, three = plans
    lib, desc = one._lib, caches[0]._desc()
    assert lib.moba_decode_attend_variant(ctypes.byref(desc), requests, hq, int(mode == "moba"), one._slots, one._umax, 0, -1) in (8, 16)

    def launch(kind, projected=None):
        p, d, st = three, caches[1]._desc(), three._stream()
        ids, pos = p.gpu_ids.data_ptr(), p.positions.data_ptr()
        union = (p._u_chunk.data_ptr(), p._u_mask.data_ptr(), p._u_count.data_ptr())
        status, b = caches[1]._status.data_ptr(), requests
        assert lib.moba_decode_step_begin(ctypes.byref(d), ids, pos, p.delta.data_ptr(), b, hq, None, None, None, p.q.data_ptr(), p.k.data_ptr(),
                                          p.v.data_ptr(), status, st) == 0
        selected = None if p.dense else p.selected.data_ptr()
        if not p.dense:
            assert lib.moba_decode_route(ctypes.byref(d), p.q.data_ptr(), ids, pos, b, hq, p.remote, p.width, p.scores.data_ptr(), selected,
                                         *union, st) == 0
        assert lib.moba_decode_attend(ctypes.byref(d), p.q.data_ptr(), ids, pos, b, hq, selected, p._slots, *union, p._umax,
                                      p._workspace.data_ptr(), p._ws_bytes, p.output.data_ptr(), p.lse.data_ptr(), status, st) == 0
    three.launch = launch
    for _ in range(steps):
        q, k, v = rnd(requests, hq, dim), rnd(requests, hk, dim), rnd(requests, hk, dim)
        a, b = one.step(q, k, v), three.step(q, k, v)
        torch.testing.assert_close(a.output.float(), b.output.float(), rtol=2.0 ** (-7 if dtype == torch.bfloat16 else -10), atol=2e-5)
        torch.testing.assert_close(a.lse, b.lse, rtol=1e-5, atol=1e-5)
        assert torch.equal(one.positions, three.positions)
        if mode == "moba":
            assert torch.equal(a.selected_blocks, b.selected_blocks) and torch.equal(one.scores, three.scores)
    for t in ("_table", "_lengths"):
        assert torch.equal(getattr(caches[0], t), getattr(caches[1], t))
    for p in plans:
        p.close()
    for sid in range(requests):
        for x, y in zip(caches[0].materialize(sid), caches[1].materialize(sid)):
            assert torch.equal(x, y)
        closed = caches[0].lengths[sid] // chunk
        assert torch.equal(caches[0]._means[sid, :closed], caches[1]._means[sid, :closed])


def twin_plans(lens, hq, hk, dim, chunk, page, mode, dtype, room, seed, k0=None, v0=None):
    """Two plans over equal caches: the first one's step is `moba_decode_step`, the second one's the entry points that it stands for."""
    import ctypes
    from moba_opt import PagedKVCache
    gen = torch.Generator().manual_seed(seed)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    k0, v0 = (torch.randn(cu[-1], hk, dim, generator=gen).to("cuda", dtype) if t is None else t for t in (k0, v0))
    plans, ids = [], list(range(len(lens)))
    for _ in range(2):
        cache = PagedKVCache(len(lens), max(lens) + room, hk, dim, page_size=page, chunk_size=chunk, dtype=dtype)
        cache.append_prefill(k0, v0, sequence_ids=ids, cu_seqlens=cu, check_finite=False)
        plans.append(cache.prepare_decode(ids, hq, topk=3, mode=mode, check_finite=False))
    one, p = plans

    def launch(kind, projected=None):
        lib, d, st, rows = p._lib, p.cache._desc(), p._stream(), len(lens)
        seqs, pos, status = p.gpu_ids.data_ptr(), p.positions.data_ptr(), p.cache._status.data_ptr()
        union = (p._u_chunk.data_ptr(), p._u_mask.data_ptr(), p._u_count.data_ptr())
        qkv, cos, sin = (None, None, None) if projected is None else (t.data_ptr() for t in projected)
        assert lib.moba_decode_step_begin(ctypes.byref(d), seqs, pos, p.delta.data_ptr(), rows, hq, qkv, cos, sin, p.q.data_ptr(), p.k.data_ptr(),
                                          p.v.data_ptr(), status, st) == 0
        selected = None if p.dense else p.selected.data_ptr()
        if not p.dense:
            assert lib.moba_decode_route(ctypes.byref(d), p.q.data_ptr(), seqs, pos, rows, hq, p.remote, p.width, p.scores.data_ptr(), selected,
                                         *union, st) == 0
        assert lib.moba_decode_attend(ctypes.byref(d), p.q.data_ptr(), seqs, pos, rows, hq, selected, p._slots, *union, p._umax,
                                      p._workspace.data_ptr(), p._ws_bytes, p.output.data_ptr(), p.lse.data_ptr(), status, st) == 0
    p.launch = launch
    return one, p


@pytest.mark.parametrize("lens,hq,hk,dim,chunk,page,mode,dtype", [
    ((63, 94), 14, 2, 64, 32, 16, "moba", torch.bfloat16),     # one row completes its chunk, the other does not
    ((63,), 14, 2, 64, 32, 16, "dense", torch.bfloat16),
    ((71, 95, 72), 6, 1, 128, 24, 7, "moba", torch.float16),   # pages across a chunk's end
    ((31, 47), 8, 4, 32, 16, 5, "moba", torch.float16),        # eight CTAs a pair
])
def test_a_new_token_without_a_page(lens, hq, hk, dim, chunk, page, mode, dtype):
    """The page of a row's new token is not mapped (a caller of the C entries without the planner): one launch and the separate ones
    report it, leave the chunk's mean and the pool alone, and give the same routes, positions, lengths and outputs."""
    import moba_opt.grouped_attention as ga
    plans = twin_plans(lens, hq, hk, dim, chunk, page, mode, dtype, 2 * chunk, 41 + dim)
    results = []
    for p in plans:
        c = p.cache
        ga.check_status()
        for sid, n in enumerate(lens):
            assert n % page, "the page exists already"
            c._table[sid, n // page] = -1
        c._means[:, :, :] = 3.0
        bits = [t.view(torch.int16) for t in (c.k_cache, c.v_cache)]     # unused pages may hold anything, NaN among it
        pools = [t.clone() for t in bits]
        gen = torch.Generator().manual_seed(5)
        q, k, v = (torch.randn(len(lens), h, dim, generator=gen).to("cuda", dtype) for h in (hq, hk, hk))
        p.stage_inputs(((q, p.q), (k, p.k), (v, p.v)))
        p.launch("step")
        with pytest.raises(RuntimeError, match="status bits"):
            ga.check_status()
        assert torch.equal(pools[0], bits[0]) and torch.equal(pools[1], bits[1])
        assert bool((c._means == 3.0).all())
        results.append([t.clone() for t in (c._table, c._lengths, p.positions, p.output, p.lse)] + ([] if p.dense else [p.selected.clone()]))
    one, separate = results
    for i in (0, 1, 2, 5)[:len(one) - 2]:
        assert torch.equal(one[i], separate[i])
    # the bounds of test_step_in_one_launch_equals_its_three_launches: neighbouring 16-bit values
    torch.testing.assert_close(one[3].float(), separate[3].float(), rtol=2.0 ** (-7 if dtype == torch.bfloat16 else -10), atol=2e-5)
    torch.testing.assert_close(one[4], separate[4], rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("mode", ["moba", "dense"])
@pytest.mark.parametrize("length", [40, 1500])       # less than a stage for each CTA of a cluster, and more
def test_a_new_token_whose_product_overflows(mode, length):
    """q . k of the new token is -inf in FP32: it has no weight, in one launch as in the separate ones."""
    hq, hk, dim = 4, 2, 64
    results = []
    for p in twin_plans((length,), hq, hk, dim, 512 if length > 512 else 32, 16, mode, torch.bfloat16, 8, 77):
        gen = torch.Generator().manual_seed(9)
        q, k, v = (torch.randn(1, h, dim, generator=gen).to("cuda", torch.bfloat16) for h in (hq, hk, hk))
        q[:, :, 0], k[:, :, 0] = 2.0 ** 70, -(2.0 ** 70)
        r = p.step(q, k, v)
        results.append((r.output.clone(), r.lse.clone()))
    (out, lse), (want, want_lse) = results
    assert bool(want.isfinite().all()) and bool(want_lse.isfinite().all())
    assert torch.equal(out, want)                    # scores of 2^70: all the weight is on one token
    torch.testing.assert_close(lse, want_lse, rtol=1e-5, atol=0)


def projected_step(p, qkv, cos, sin):
    """One step from the fused projection, as a model session drives it; returns whether it was one launch (plans that route)."""
    plan = p.plan_step()
    p.send_delta(plan)
    p._u_count.fill_(-7)                       # the one-launch form leaves the union lists alone
    p.launch("step", (qkv, cos, sin))
    p.commit_step(plan)
    return p.dense or bool((p._u_count == -7).all())


@pytest.mark.parametrize("lens,hq,hk,dim,chunk,page,mode,offset,one_launch", [
    ((61, 94, 33), 14, 2, 64, 32, 16, "moba", 0, True),
    ((20, 47), 8, 2, 32, 16, 5, "dense", 0, True),
    ((70, 95), 6, 1, 96, 24, 7, "moba", 0, True),
    ((63, 40, 55, 90), 8, 2, 128, 32, 16, "moba", 0, True),
    ((63, 40), 20, 2, 128, 32, 16, "dense", 0, True),      # two head blocks
    ((45, 61), 4, 2, 24, 16, 8, "moba", 0, False),         # half a head is not whole 16-byte units
    ((61, 94), 14, 2, 64, 32, 16, "moba", 4, False),       # a projection 8 bytes off
])
def test_step_from_a_projection_equals_its_three_launches(lens, hq, hk, dim, chunk, page, mode, offset, one_launch):
    """Rotary embedding and split of several rows inside the one launch, or in front of the separate ones where it cannot be taken."""
    dtype, rows, width = torch.bfloat16, len(lens), (hq + 2 * hk) * dim
    one, separate = twin_plans(lens, hq, hk, dim, chunk, page, mode, dtype, 2 * chunk, 13 + dim)
    gen = torch.Generator().manual_seed(dim + hq)
    for _ in range(chunk + 3):
        flat = torch.randn(rows * width + offset, generator=gen).to("cuda", dtype)
        qkv = flat[offset:].view(rows, width)
        angle = torch.rand(rows, dim, generator=gen) * 6.3
        cos, sin = angle.cos().to("cuda", dtype), angle.sin().to("cuda", dtype)
        took = projected_step(one, qkv, cos, sin)
        projected_step(separate, qkv, cos, sin)
        assert mode == "dense" or took == one_launch
        for name in ("q", "k", "v", "positions"):
            assert torch.equal(getattr(one, name), getattr(separate, name)), name
        if mode == "moba":
            assert torch.equal(one.selected, separate.selected) and torch.equal(one.scores, separate.scores)
        # the bounds of test_step_in_one_launch_equals_its_three_launches
        torch.testing.assert_close(one.output.float(), separate.output.float(), rtol=2.0 ** -7, atol=2e-5)
        torch.testing.assert_close(one.lse, separate.lse, rtol=1e-5, atol=1e-5)
    a, b = one.cache, separate.cache
    assert torch.equal(a._table, b._table) and torch.equal(a._lengths, b._lengths)
    for p in (one, separate):
        p.close()
    for sid in range(rows):
        for x, y in zip(a.materialize(sid), b.materialize(sid)):
            assert torch.equal(x, y)
        closed = a.lengths[sid] // chunk
        assert closed and torch.equal(a._means[sid, :closed], b._means[sid, :closed])


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("rows,hq,hk,dim,dtype", [
    (1, 8, 2, 64, torch.bfloat16),
    (2, 6, 1, 128, torch.float16),
    (4, 40, 2, 128, torch.bfloat16),                       # eight CTAs a pair, two head blocks
    (3, 4, 1, 32, torch.bfloat16),
])
def test_a_step_over_values_that_are_not_finite(rows, hq, hk, dim, dtype, bad):
    """Such a V (of a caller that switched the check off) reaches the heads that attend its chunk and no other one, cached or new,
    in the one-launch step as in the separate ones; every other value keeps its bits."""
    chunk, chunks, poisoned = 100, 6, 2
    length = chunks * chunk + 41
    gen = torch.Generator().manual_seed(411)
    rnd = lambda *shape: torch.randn(*shape, generator=gen).to("cuda", dtype)
    k, v = rnd(length, hk, dim), rnd(length, hk, dim)
    k[:, :, :chunks] = 0
    for c in range(chunks):
        k[c * chunk:(c + 1) * chunk, :, c] = 8             # chunk c is the best match of a query along axis c
    turns = [(rnd(rows, hq, dim), rnd(rows, hk, dim), rnd(rows, hk, dim)) for _ in range(3)]
    for q, _, _ in turns:
        for h in range(hq):
            q[:, h, h % chunks] = 40
    seen = {}
    for value in (1.0, bad):
        vv = v.clone()
        vv[poisoned * chunk + 33, :, 5] = value
        one, separate = twin_plans((length,) * rows, hq, hk, dim, chunk, 7, "moba", dtype, 8, 0, k.repeat(rows, 1, 1), vv.repeat(rows, 1, 1))
        seen[value] = []
        for turn, (q, kn, vn) in enumerate(turns):
            vn = vn.clone()
            if turn == 1:
                vn[:, :, 7] = value                        # the new token's
            a, b = one.step(q, kn, vn), separate.step(q, kn, vn)
            assert torch.equal(a.selected_blocks, b.selected_blocks) and torch.equal(a.output.isfinite(), b.output.isfinite())
            seen[value].append((a.output.clone(), a.lse.clone(), a.selected_blocks.clone()))
    for turn, ((good, lse, picks), (spoiled, lse_spoiled, _)) in enumerate(zip(seen[1.0], seen[bad])):
        reads = (picks == poisoned).any(-1)
        assert reads.any() and not reads.all()
        assert bool(good.isfinite().all()) and torch.equal(lse, lse_spoiled)
        wrong = torch.zeros_like(good, dtype=torch.bool)
        wrong[..., 5] |= reads
        if turn > 0:
            wrong[..., 7] = True
        assert torch.equal(spoiled.isfinite(), ~wrong)
        assert torch.equal(good[~wrong], spoiled[~wrong])
        if bad == bad:                                     # an infinity stays one, of its sign
            assert (spoiled[wrong] == bad).all()
