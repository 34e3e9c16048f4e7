"""CPU tests of the page allocator and the incremental decode lease.  They pin the behaviours the
reference's tests pin (tests/test_cache_layout.py:13-68, tests/test_prepared_layout.py:6-30):
atomic planning, stale plans, LIFO page reuse, page math for non-dividing sizes, and equivalence of
the incremental lease with the transactional allocator."""
import copy
import pickle
import random
from dataclasses import FrozenInstanceError, replace

import pytest

from moba_opt.cache_layout import AppendPlan, IncrementalLayout, PageAllocator


def snapshot(a):
    return a.tables, a.lengths, a.free_pages, a.version


def test_planning_is_side_effect_free_and_commit_is_versioned():
    a = PageAllocator(2, 17, 3, 12, 4)
    before = snapshot(a)
    plan = a.plan_append([1, 0], [5, 7])
    assert snapshot(a) == before
    assert plan.token_sequences == (1,) * 5 + (0,) * 7
    assert plan.token_positions == tuple(range(5)) + tuple(range(7))
    assert plan.completed_chunks == ((1, 0), (0, 0))
    a.commit(plan)
    assert a.lengths == (7, 5)
    assert a.tables[1][:2] == (0, 1) and a.tables[0][:3] == (2, 3, 4)   # page 0 is handed out first
    with pytest.raises(RuntimeError, match="stale"):
        a.commit(plan)


def test_released_pages_are_reused_last_in_first_out():
    a = PageAllocator(3, 12, 3, 4, 4)
    a.commit(a.plan_append([0, 1], [6, 3]))
    a.reset([0])
    a.commit(a.plan_append([2], [6]))
    assert a.tables[2][:2] == (1, 0)
    assert a.tables[1][0] == 2
    assert len(a.free_pages) == 1


@pytest.mark.parametrize("ids,counts", [([1], [1]), ([0], [20]), ([0, 0], [1, 1]), ([2], [1]), ([0], [0]), ([0], [True]),
                                        ([0.5], [1]), ([], [])])
def test_rejected_appends_leave_state_untouched(ids, counts):
    a = PageAllocator(2, 12, 3, 2, 4)
    a.commit(a.plan_append([0], [4]))
    before = snapshot(a)
    with pytest.raises(ValueError):
        a.plan_append(ids, counts)
    assert snapshot(a) == before


def test_pool_exhaustion_message():
    a = PageAllocator(2, 12, 3, 2, 4)
    a.commit(a.plan_append([0], [4]))
    with pytest.raises(ValueError, match="pool exhausted"):
        a.plan_append([1], [1])
    with pytest.raises(ValueError, match="max_seq_len"):
        a.plan_append([0], [20])


def test_completed_chunks_follow_logical_positions():
    a = PageAllocator(1, 20, 3, 7, 4)
    a.commit(a.plan_append([0], [3]))
    p = a.plan_append([0], [6])
    assert p.completed_chunks == ((0, 0), (0, 1))
    a.commit(p)
    assert a.plan_append([0], [1]).completed_chunks == ()


@pytest.mark.parametrize("page", [1, 3, 7, 16, 31, 48])
def test_page_accounting_for_sizes_that_do_not_divide(page):
    a = PageAllocator(2, 65, page, 2 * ((65 + page - 1) // page), 24)
    a.commit(a.plan_append([0, 1], [65, 33]))
    owned = [x for row in a.tables for x in row if x >= 0]
    assert len(owned) == len(set(owned))
    assert len(owned) + len(a.free_pages) == a.num_pages
    a.reset([0, 1])
    assert len(a.free_pages) == a.num_pages and a.lengths == (0, 0)


def test_int32_capacity_guard():
    with pytest.raises(ValueError, match="int32"):
        PageAllocator(1, 2 ** 30, 16, 4, 8)
    with pytest.raises(ValueError, match="int32"):
        PageAllocator(1, 64, 2 ** 16, 2 ** 15, 8)


@pytest.mark.parametrize("page", [1, 3, 7, 16])
def test_incremental_lease_equals_transactional_allocator(page):
    old = PageAllocator(3, 41, page, 3 * ((41 + page - 1) // page), 8)
    old.commit(old.plan_append([1, 0], [5, 7]))
    old.reset([1])
    fast = IncrementalLayout(old, [2, 0, 1])
    for _ in range(30):
        plan = fast.plan()
        before = (tuple(map(tuple, fast.tables)), tuple(fast.lengths), tuple(fast.free))
        assert fast.plan() == plan
        assert before == (tuple(map(tuple, fast.tables)), tuple(fast.lengths), tuple(fast.free))
        fast.commit(plan)
        old.commit(old.plan_append([2, 0, 1], [1, 1, 1]))
        assert tuple(map(tuple, fast.tables)) == old.tables
        assert tuple(fast.lengths) == old.lengths and tuple(fast.free) == old.free_pages
    fast.publish(old)
    assert old.lengths == (37, 30, 30)
    with pytest.raises(RuntimeError, match="stale"):
        fast.commit(plan)


def test_incremental_failures_do_not_mutate():
    old = PageAllocator(2, 4, 2, 1, 2)
    old.commit(old.plan_append([0], [2]))
    fast = IncrementalLayout(old, [0, 1])
    with pytest.raises(ValueError, match="pool exhausted"):
        fast.plan()
    assert fast.lengths == [2, 0] and fast.free == []
    old = PageAllocator(1, 1, 1, 1, 1)
    old.commit(old.plan_append([0], [1]))
    with pytest.raises(ValueError, match="max_seq_len"):
        IncrementalLayout(old, [0]).plan()


@pytest.mark.parametrize("page", [3, 4, 7])
def test_plan_without_token_lists_is_the_same_plan(page):
    """A whole-prompt append (append_prefill) plans without the per-token (sequence, position) lists; everything else
    of the plan - tables, lengths, pool, completed chunks - is what the full plan gives."""
    a = PageAllocator(3, 40, page, 40, 8)
    a.commit(a.plan_append([2], [5]))
    full = a.plan_append([0, 2, 1], [13, 9, 1])
    light = a.plan_append([0, 2, 1], [13, 9, 1], tokens=False)
    assert light.token_sequences == () and light.token_positions == ()
    assert len(full.token_sequences) == 23
    for field in ("version", "tables", "lengths", "free_pages", "completed_chunks"):
        assert getattr(full, field) == getattr(light, field)
    a.commit(light)
    assert a.lengths == (13, 1, 14)


class EagerAllocator:
    """The allocator's contract in its plainest form: every plan and every state is a copy of everything."""

    def __init__(self, sequences, width, page, pages):
        self.page = page
        self.tables, self.lengths = ((-1,) * width,) * sequences, (0,) * sequences
        self.free_pages = tuple(range(pages - 1, -1, -1))

    def append(self, ids, counts):
        tables, lengths, pool = [list(row) for row in self.tables], list(self.lengths), list(self.free_pages)
        for sid, n in zip(ids, counts):
            for logical in range(-(-lengths[sid] // self.page), -(-(lengths[sid] + n) // self.page)):
                tables[sid][logical] = pool.pop()
            lengths[sid] += n
        return tuple(map(tuple, tables)), tuple(lengths), tuple(pool)

    def reset(self, ids):
        tables, lengths, pool = list(self.tables), list(self.lengths), list(self.free_pages)
        for sid in ids:
            pool += [p for p in tables[sid] if p >= 0]
            tables[sid], lengths[sid] = (-1,) * len(tables[sid]), 0
        return tuple(tables), tuple(lengths), tuple(pool)


def shown(x):
    return x.tables, x.lengths, x.free_pages


@pytest.mark.parametrize("seed", range(6))
def test_plans_are_snapshots_whatever_the_allocator_does_next(seed):
    """Plans hold what an append changes and build tables and pool late; what they show, and what the allocator shows, is what copies
    made at once would: read before or after the commit, after later commits, resets and leases, or never."""
    rng = random.Random(seed)
    a, plain = PageAllocator(3, 40, 3, 30, 4), EagerAllocator(3, 14, 3, 30)
    kept = [(a.tables, plain.tables)]
    for _ in range(60):
        ids = rng.sample(range(3), rng.randint(1, 3))
        step = rng.randrange(4)
        if step == 0:
            a.reset(ids)
            plain.tables, plain.lengths, plain.free_pages = plain.reset(ids)
        elif step == 1 and max(a.lengths) < 40 and len(a.free_pages) >= 3:
            lease = IncrementalLayout(a, ids)
            lease.commit(lease.plan())
            lease.publish(a)
            plain.tables, plain.lengths, plain.free_pages = plain.append(ids, [1] * len(ids))
        else:
            counts = [rng.randint(1, 9) for _ in ids]
            try:
                plan, other = a.plan_append(ids, counts), a.plan_append(ids[:1], counts[:1], tokens=False)
            except ValueError:
                continue
            want, unused = plain.append(ids, counts), plain.append(ids[:1], counts[:1])
            if rng.random() < 0.3:
                assert shown(plan) == want
            if rng.random() < 0.5:
                kept.append((other, unused))
            if rng.random() < 0.7:
                a.commit(plan)
                plain.tables, plain.lengths, plain.free_pages = want
            kept.append((plan, want))
        assert shown(a) == shown(plain)
        kept.append((a.tables, plain.tables))
        if len(kept) > 12:
            got, want = kept.pop(rng.randrange(len(kept)))
            assert (shown(got) if isinstance(got, AppendPlan) else got) == want
    for got, want in kept:
        assert (shown(got) if isinstance(got, AppendPlan) else got) == want


def test_plans_and_allocators_are_values():
    """A plan is a frozen dataclass of its fields, and commit takes any plan of the present version; clones, copies and pickles of an
    allocator stand for themselves, and a snapshot that nothing has changed is not built again."""
    a = PageAllocator(2, 20, 3, 14, 4)
    a.commit(a.plan_append([1], [4]))
    plan, same, first = (a.plan_append([0, 1], [7, 3]) for _ in range(3))
    assert plan == same and hash(plan) == hash(same) and repr(plan) == repr(same) and "tables=((2, 3, 4" in repr(plan)
    with pytest.raises(FrozenInstanceError):
        plan.lengths = ()
    whole = AppendPlan(plan.version, plan.tables, plan.lengths, plan.free_pages, plan.token_sequences, plan.token_positions,
                       plan.completed_chunks, plan.page_edits)
    assert whole == plan == copy.copy(same) == pickle.loads(pickle.dumps(first)) == replace(first, page_edits=first.page_edits)
    twins = [a.clone(), copy.copy(a), copy.deepcopy(a), pickle.loads(pickle.dumps(a))]
    before = snapshot(a)
    for twin, made in zip(twins, (whole, plan, a.plan_append([0, 1], [7, 3]), twins[3].plan_append([0, 1], [7, 3]))):
        assert snapshot(twin) == before
        twin.commit(made)                                  # another allocator's plan among them
        assert shown(twin) == shown(plan) and snapshot(a) == before
        twin.reset([0])
        assert snapshot(a) == before
    assert a.tables is a.tables
    a.commit(a.plan_append([0], [1]))
    assert a.tables is a.tables and a.tables[1] is before[0][1]     # the row that did not change
    with pytest.raises(RuntimeError, match="stale"):
        a.commit(plan)


def test_a_plan_shows_the_next_state_until_the_allocator_moves_on():
    """A plan holds what an append changes; its tables and pool are the next state's before and after the commit, and are
    refused once another call has changed the allocator."""
    a = PageAllocator(2, 20, 3, 14, 4)
    a.commit(a.plan_append([1], [4]))
    first, second = a.plan_append([0, 1], [7, 3]), a.plan_append([0], [2])
    want = (first.tables, first.free_pages)
    assert want[0][0][:3] == (2, 3, 4) and want[0][1][:3] == (0, 1, 5) and len(want[1]) == 8
    a.commit(first)
    assert (a.tables, a.free_pages) == want == (first.tables, first.free_pages)
    for stale in (lambda: a.commit(second), lambda: second.tables, lambda: second.free_pages, lambda: a.reset([0]) or first.tables):
        with pytest.raises(RuntimeError, match="stale"):
            stale()
    other = PageAllocator(2, 20, 3, 14, 4)
    with pytest.raises(RuntimeError, match="stale"):      # a plan of another allocator
        other.commit(PageAllocator(2, 20, 3, 14, 4).plan_append([0], [1]))


@pytest.mark.parametrize("ids,counts", [((2,), (1,)), ((0, 2), (3, 5)), ((1, 0, 2), (20, 40, 4)), ((1, 0, 2), (20, 40, 5)), ((1,), (700,))])
def test_rows_of_an_append_in_both_forms(ids, counts):
    """Up to 64 tokens and more: the ids and positions that a full plan lists."""
    from moba_opt.kv_cache import token_rows
    a = PageAllocator(3, 1000, 7, 500, 16)
    a.commit(a.plan_append([0, 2], [11, 30]))
    plan = a.plan_append(ids, counts)
    rows = token_rows(ids, counts, a.lengths)
    assert all(isinstance(r, tuple) == (sum(counts) <= 64) for r in rows)
    assert [tuple(int(x) for x in r) for r in rows] == [plan.token_sequences, plan.token_positions]
