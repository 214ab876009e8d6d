"""The memory kept of a freed database is given back to whichever allocation of the engine on
the device needs it: another context's import (into the block itself, or into what it frees),
a served query of the same or of another context, a reply's workspaces.  The device is filled by one allocation that leaves less free
than each of them needs."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import random_db, random_query

pytestmark = pytest.mark.gpu

N, M, LEFT = 1024, 2, 140 << 20


@pytest.fixture
def full_device(engine):
    """fill(): the device has at most LEFT bytes free until the test ends."""
    torch = pytest.importorskip("torch")
    held = []

    def fill():
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        held.append(torch.empty(torch.cuda.mem_get_info()[0] - LEFT, dtype=torch.uint8, device="cuda"))
        assert torch.cuda.mem_get_info()[0] <= LEFT

    yield fill
    held.clear()
    torch.cuda.empty_cache()


def keep_spare(ctx, b):
    """Leaves ctx with the 328 MB of a freed database."""
    torch = pytest.importorskip("torch")
    F = 20000
    ctx.import_db(torch.zeros(F * 64, dtype=torch.uint8, device="cuda"), F, 64, 1, b).free()


@pytest.mark.parametrize("F", [9900, 13000])  # 162 MB of words: too few for the block; 213 MB
def test_import_of_another_context(engine, oracle, full_device, F):
    torch = pytest.importorskip("torch")
    b, L = oracle.bits_per_coeff(N, M, 40), 64
    elems = random_db(150, F, L)
    dev = torch.from_numpy(elems).cuda()
    with engine.Context(N, M) as first, engine.Context(N, M) as second:
        keep_spare(first, b)
        full_device()
        d = second.import_db(dev, F, L, 1, b)
        few = 50
        want = oracle.import_db(elems[:few * L], few, L, 1, b, N, M)
        assert np.array_equal(d.export()[:want.size], want)
        d.free()
        again = first.import_db(dev, F, L, 1, b)  # second's block now, through first
        assert np.array_equal(again.export()[:want.size], want)


@pytest.mark.parametrize("own", [True, False])
def test_served_query(engine, oracle, full_device, own):
    """A 213 MB query of a small database on a grid that is mostly empty."""
    n, F, L = [6500], 60, 500
    b = oracle.bits_per_coeff(N, M, n[0])
    q = random_query(151, n, N, M, oracle.moduli(M))
    with engine.Context(N, M) as serving, engine.Context(N, M) as other:
        d = serving.import_db(random_db(152, F, L), F, L, 1, b)
        want = oracle.reply(d.export(), F, 1, [F], q[:F * 2 * M * N], b, N, M)
        with engine.Server([serving], 4 << 30) as server:
            keep_spare(serving if own else other, b)
            full_device()
            replies = np.zeros(want.size, dtype=np.uint64)
            assert server.wait(server.submit(d, n, q, replies))[0] == 1
        # 6,440 empty slots subtract what p they can
        p = np.array(oracle.moduli(M), dtype=np.uint64)
        w = want.reshape(2, M, N).copy()
        for _ in range(8):
            w = np.where(w >= p[None, :, None], w - p[None, :, None], w)
        assert np.array_equal(replies.reshape(2, M, N), w)


def test_workspaces_of_a_recursive_reply(engine, oracle, full_device):
    """Level replies and the next level's database, 49 and 147 MB."""
    n, F, L = [2, 1500], 3000, 300
    b = oracle.bits_per_coeff(N, M, n[0])
    q = random_query(153, n, N, M, oracle.moduli(M))
    torch = pytest.importorskip("torch")
    with engine.Context(N, M) as ctx, engine.Context(N, M) as other:
        d = ctx.import_db(random_db(154, F, L), F, L, 1, b)
        dq = torch.from_numpy(q.view(np.int64)).cuda()
        want = ctx.reply(d, n, dq)
        keep_spare(other, b)
        with engine.Context(N, M) as fresh:
            d2 = fresh.import_db(random_db(154, F, L), F, L, 1, b)
            full_device()
            assert np.array_equal(fresh.reply(d2, n, dq), want)


def test_at_most_one_gib_per_device(engine, oracle):
    torch = pytest.importorskip("torch")
    b, F = oracle.bits_per_coeff(N, M, 40), 40000  # 655 MB of words each
    elems = torch.zeros(F * 64, dtype=torch.uint8, device="cuda")
    size = F * M * N * 8
    ctxs = [engine.Context(N, M) for _ in range(3)]
    dbs = [c.import_db(elems, F, 64, 1, b) for c in ctxs]
    torch.cuda.synchronize()
    free = [torch.cuda.mem_get_info()[0]]
    for d in dbs:
        d.free()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[3] - free[0] >= 2 * size  # one block is kept, not three
    for c in ctxs:
        c.close()
    assert torch.cuda.mem_get_info()[0] - free[0] >= 3 * size
