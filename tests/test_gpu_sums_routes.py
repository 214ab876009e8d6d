"""Levels that residue sums reply to, by the launches that they take: a level cut into runs is
two (reply_sum_kernel and reply_finish_kernel), one run per column one, and a repeat slot by
slot one a level more.  Words that the sums cannot decide in the first run, in the middle, at
the ends of the prefix and in the exact tail; columns with stretches of all-zero elements.
Integer work: bit-exact, no tolerance."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from helpers import random_db, random_query, shapes

pytestmark = pytest.mark.gpu


def launches(ctx, call):
    before = ctx.launch_count
    result = call()
    return result, ctx.launch_count - before


# N, m, n levels, alpha, nb elements, element bytes, launches of a reply
SHAPES = [
    (512, 1, [600], 1, 600, 200, 2),        # the fewest slots of a lone column
    (512, 1, [605], 1, 605, 200, 2),        # slots past the last tile
    (512, 1, [607], 2, 1200, 200, 2),       # a few empty slots, aggregated elements
    (512, 1, [1500], 1, 700, 200, 2),       # more empty slots than others
    (512, 7, [613], 1, 613, 200, 2),        # seven moduli
    (8192, 2, [600], 1, 600, 5000, 2),      # the largest degree
    (1024, 1, [602], 1, 602, 9500, 2),      # five columns in pairs, runs
    (512, 1, [640], 1, 640, 3200, 2),       # four columns in pairs, runs
    (512, 1, [700], 1, 700, 2500, 2),       # three columns a CTA, runs
    (8192, 4, [100], 1, 100, 8000, 1),      # a lone column in one run
    (8192, 2, [130], 1, 130, 110000, 1),    # three columns a CTA, one run
    (2048, 2, [24, 70], 1, 1670, 900, 3),   # pairs, one run of one tile before the tail; a level by slot
    (512, 2, [128, 301], 1, 38500, 60, 3),  # four columns a CTA, one run, a last block of one column
    (512, 2, [20, 700], 1, 14000, 60, 4),   # one run, then a level in runs
    (1024, 1, [650, 12], 1, 7790, 100, 4),  # runs of a partial last group, then a level by slot
]


@pytest.mark.parametrize("N,m,n,alpha,F,L,count", SHAPES)
def test_routes_equal_oracle(engine, oracle, N, m, n, alpha, F, L, count):
    b, P = shapes(N, m, n, alpha, L, oracle)
    q = random_query(162, n, N, m, oracle.moduli(m))
    with engine.Context(N, m) as ctx:
        d = ctx.import_db(random_db(161, F, L), F, L, alpha, b)
        want = oracle.reply(d.export(), -(-F // alpha), P, n, q, b, N, m)
        got, took = launches(ctx, lambda: ctx.reply(d, n, q))
        assert np.array_equal(got, want)
        assert took == count


# Slots of level 1 at both ends and in the middle of the prefix and of the tail.
UNDECIDED = [
    (512, 1, [605], 605, 200, 2, 1, (0, 300, 591, 592, 604)),           # runs, one column
    (512, 1, [700], 700, 2500, 2, 1, (0, 71, 400, 687, 688, 699)),      # runs, three columns
    (8192, 4, [100], 100, 8000, 1, 1, (0, 40, 87, 88, 99)),             # one run, one column
    (8192, 2, [130], 130, 110000, 1, 1, (0, 64, 111, 112, 129)),        # one run, three columns
    (2048, 2, [24, 70], 1670, 900, 3, 3, (0, 7, 8, 23)),                # one run, pairs
    (512, 2, [128, 301], 38500, 60, 3, 3, (5, 111, 127)),               # one run, four columns
]


@pytest.mark.parametrize("N,m,n,F,L,count,repeat,slots", UNDECIDED)
def test_undecided_words_anywhere(engine, oracle, N, m, n, F, L, count, repeat, slots):
    b, P = shapes(N, m, n, 1, L, oracle)
    ordinary = random_query(171, n, N, m, oracle.moduli(m))
    p = oracle.moduli(m)[m - 1]
    with engine.Context(N, m) as ctx:
        d = ctx.import_db(random_db(170, F, L), F, L, 1, b)
        imp = d.export()
        plain = oracle.reply(imp, F, P, n, ordinary, b, N, m)
        for k, slot in enumerate(slots):
            q = ordinary.reshape(sum(n), 2, m, N).copy()
            q[slot, k % 2, m - 1, (N - 1, 0, 129)[k % 3]] = (p, 2**64 - 1, p + 1, 2**61, 2**63)[k % 5]
            q = q.reshape(-1)
            want = oracle.reply(imp, F, P, n, q, b, N, m)
            got, took = launches(ctx, lambda: ctx.reply(d, n, q))
            assert np.array_equal(got, want), slot
            assert took == count + repeat, slot
            got, took = launches(ctx, lambda: ctx.reply(d, n, ordinary))
            assert np.array_equal(got, plain) and took == count


@pytest.mark.parametrize("kind", ["zero words", "zero query", "constant words", "arbitrary words"])
@pytest.mark.parametrize("N,m,n,F,L", [(512, 1, [605], 605, 200), (512, 1, [700], 700, 2500),
                                       (8192, 2, [130], 130, 110000), (512, 2, [128, 301], 38500, 60)])
def test_whole_queries_of_unusual_words(engine, oracle, N, m, n, F, L, kind):
    """In waves of CTAs the later ones see the stop flag of the first; the next reply does not."""
    b, P = shapes(N, m, n, 1, L, oracle)
    ordinary = random_query(176, n, N, m, oracle.moduli(m))
    elems = random_db(175, F, L)
    w = ordinary.reshape(sum(n), 2, m, N).copy()
    if kind == "zero words":
        w[:, :, :, ::2] = 0
    elif kind == "zero query":
        w[:] = 0
    elif kind == "constant words":
        w[:] = w[0]
        elems = np.tile(elems[:L], F)  # the same term in every slot
    else:
        w = random_query(177, n, N, m, oracle.moduli(m), reduced=False)
    q = w.reshape(-1)
    with engine.Context(N, m) as ctx:
        d = ctx.import_db(elems, F, L, 1, b)
        imp = d.export()
        for query in (q, ordinary, q):
            assert np.array_equal(ctx.reply(d, n, query), oracle.reply(imp, F, P, n, query, b, N, m))


def test_noalloc_undecided(engine, oracle):
    torch = pytest.importorskip("torch")
    N, m, n, F, L = 512, 1, [605], 605, 200
    b, P = shapes(N, m, n, 1, L, oracle)
    fn = engine.lib().xpir_b200_reply_noalloc
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint32, ctypes.POINTER(ctypes.c_uint32),
                   ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint64, ctypes.POINTER(ctypes.c_uint64)]
    with engine.Context(N, m) as ctx:
        d = ctx.import_db(random_db(173, F, L), F, L, 1, b)
        for slot in (None, 3, 591, 600):
            q = random_query(174, n, N, m, oracle.moduli(m))
            if slot is not None:
                q[slot * 2 * m * N + 17] = 2**62
            want = oracle.reply(d.export(), F, P, n, q, b, N, m)
            qd = torch.from_numpy(q.view(np.int64)).cuda()
            out = torch.full((want.size,), -1, dtype=torch.int64, device="cuda")
            status, took = launches(ctx, lambda: fn(ctx.handle, d.handle, 1, (ctypes.c_uint32 * 1)(*n), qd.data_ptr(),
                                                    out.data_ptr(), out.numel() * 8, ctypes.byref(ctypes.c_uint64())))
            assert status == engine.OK
            assert np.array_equal(out.cpu().numpy().view(np.uint64), want)
            assert took == (2 if slot is None else 3)


# All-zero elements import to words 0 and p.  Where the database holds a hint, eight of them
# send it slot by slot; a context's 1,023rd database holds none, and the sums tell by
# themselves: ten at the end of a column are decided from further back, a hundred in a row or
# sixty up to the end are not (None: either way, the reply is the same).
@pytest.mark.parametrize("zeros,with_hint,without", [
    (range(0, 7), 2, 2), (range(0, 8), 1, None), (range(693, 700), 2, 2), (range(690, 700), 1, 2),
    (range(200, 300), 1, 3), (range(640, 700), 1, 3), (range(0, 700, 10), 1, 2), (range(0, 700, 2), 1, None),
    (range(700), 1, 3)])
def test_all_zero_elements(engine, oracle, zeros, with_hint, without):
    N, m, n, F, L = 512, 1, [700], 700, 200
    b, P = shapes(N, m, n, 1, L, oracle)
    elems = random_db(181, F, L).reshape(F, L)
    elems[list(zeros)] = 0
    elems = elems.reshape(-1)
    q = random_query(182, n, N, m, oracle.moduli(m))
    with engine.Context(N, m) as ctx:
        d = ctx.import_db(elems, F, L, 1, b)
        want = oracle.reply(d.export(), F, P, n, q, b, N, m)
        got, took = launches(ctx, lambda: ctx.reply(d, n, q))
        assert np.array_equal(got, want)
        assert took == with_hint
        small = random_db(183, 1, L)
        held = [ctx.import_db(small, 1, L, 1, b) for _ in range(1021)]
        d2 = ctx.import_db(elems, F, L, 1, b)
        got, took = launches(ctx, lambda: ctx.reply(d2, n, q))
        assert np.array_equal(got, want)
        assert took == without or without is None
        for h in held:
            h.free()
