"""A query that the residue sums cannot decide is repeated slot by slot by itself: the other
queries of its batch are not.  Integer work: bit-exact, no tolerance."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import random_db, random_query, shapes

pytestmark = pytest.mark.gpu

N, M = 512, 1


def launches(ctx, items, use_graph):
    before = ctx.launch_count
    ctx.reply_batch(items, use_graph=use_graph)
    return ctx.launch_count - before


@pytest.mark.parametrize("use_graph", [False, True])
def test_other_grids_are_not_repeated(engine, oracle, use_graph):
    """Three grids, two queries each, cut into runs (two launches a grid); an undecided query
    adds one launch, for its grid alone."""
    torch = pytest.importorskip("torch")
    F, L, grids = 700, 500, ([700], [703], [710])
    b, P = shapes(N, M, grids[0], 1, L, oracle)
    with engine.Context(N, M) as ctx:
        d = ctx.import_db(random_db(110, F, L), F, L, 1, b)
        imp = d.export()
        items, per = [], []
        for k, n in enumerate(grids * 2):
            versions = []
            for bad in (False, True):
                q = random_query(111 + k, n, N, M, oracle.moduli(M))
                if bad and k == 4:
                    q[690 * 2 * M * N + 7] = 2**63
                versions.append((q, oracle.reply(imp, F, P, n, q, b, N, M)))
            per.append(versions)
            items.append((d, n, torch.empty(versions[0][0].size, dtype=torch.int64, device="cuda"),
                          torch.empty(versions[0][1].size, dtype=torch.int64, device="cuda")))
        counts = []
        for bad in (0, 0, 1, 1, 0):
            for (_, _, q, out), versions in zip(items, per):
                q.copy_(torch.from_numpy(versions[bad][0].view(np.int64)))
                out.fill_(-1)
            torch.cuda.synchronize()
            counts.append(launches(ctx, items, use_graph))
            for (_, _, _, out), versions in zip(items, per):
                assert np.array_equal(out.cpu().numpy().view(np.uint64), versions[bad][1])
        assert counts == [6, 6, 7, 7, 6]


def test_more_queries_than_flags(engine, oracle):
    """1,030 queries of one grid, undecided ones first, last and between."""
    torch = pytest.importorskip("torch")
    n, F, L, count, bad = [24], 24, 300, 1030, (0, 511, 1022, 1023, 1029)
    b, P = shapes(N, M, n, 1, L, oracle)
    with engine.Context(N, M) as ctx:
        d = ctx.import_db(random_db(120, F, L), F, L, 1, b)
        imp = d.export()
        qs = [random_query(121 + k, n, N, M, oracle.moduli(M)) for k in range(8)]
        want = [oracle.reply(imp, F, P, n, q, b, N, M) for q in qs]
        dq = [torch.from_numpy(q.view(np.int64)).cuda() for q in qs]
        odd = {}
        for i in bad:
            q = qs[i % 8].copy()
            q[-1 - i] = 2**64 - 1 - i
            odd[i] = (torch.from_numpy(q.view(np.int64)).cuda(), oracle.reply(imp, F, P, n, q, b, N, M))
        out = torch.full((count, want[0].size), -1, dtype=torch.int64, device="cuda")
        items = [(d, n, odd[i][0] if i in odd else dq[i % 8], out[i]) for i in range(count)]
        assert launches(ctx, items, False) == 2  # one of sums, one slot by slot
        got = out.cpu().numpy().view(np.uint64)
        for i in range(count):
            assert np.array_equal(got[i], odd[i][1] if i in odd else want[i % 8]), i
