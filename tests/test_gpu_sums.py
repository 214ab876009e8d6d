"""Replies by residue sums with an exact tail (xpir_b200/csrc/reply_sum.cu) against the
oracle, at the sizes where the path can go wrong: slot counts around the tail, the tile and
the runs, partial and idle groups at every level, and words the sums cannot decide (which
must come out of the slot-by-slot kernel instead).  Integer work: bit-exact, no tolerance."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from helpers import random_db, random_query, shapes

pytestmark = pytest.mark.gpu

# N, m, n levels, alpha, nb elements, element bytes
SHAPES = [
    (512, 1, [400], 1, 400, 200),        # the fewest slots of a lone column, one poly
    (512, 1, [405], 1, 405, 200),        # slots past the last tile
    (512, 1, [1500], 1, 402, 200),       # a grid larger than the database
    (512, 7, [431], 1, 431, 200),        # seven moduli
    (1024, 1, [1000], 1, 1000, 7000),    # several runs, an odd number of columns
    (1024, 2, [700, 3], 1, 1800, 900),   # runs, three groups, the last one partial
    (1024, 3, [100, 40], 1, 3950, 300),  # one run per column, a partial last group
    (2048, 2, [61, 60], 1, 3600, 4000),  # short chains of many columns
    (1024, 1, [70, 60], 2, 500, 500),    # 4 of 60 first-level groups with data
    (1024, 1, [6, 10, 9], 1, 150, 300),  # idle elements inside, after and between second-level groups
    (1024, 1, [6, 10, 9], 1, 180, 300),  # 30 live of 90: the second level's groups are whole
    (1024, 2, [5, 8, 3, 4], 1, 27, 300),  # four levels
    (1024, 1, [700], 1, 700, 5200),      # three columns per CTA, several runs
    (512, 2, [700, 1], 3, 2100, 2500),   # the same with two moduli and aggregation
    (512, 2, [133, 300], 1, 39870, 60),  # four columns per CTA, a partial last group
    (512, 2, [128, 301], 1, 38528, 60),  # four columns per CTA, three of the last block empty
]


@pytest.mark.parametrize("N,m,n,alpha,F,L", SHAPES)
def test_sums_equal_oracle(engine, oracle, N, m, n, alpha, F, L):
    b, P = shapes(N, m, n, alpha, L, oracle)
    q = random_query(32, n, N, m, oracle.moduli(m))
    with engine.Context(N, m) as ctx:
        d = ctx.import_db(random_db(31, F, L), F, L, alpha, b)
        imp = d.export()
        want = oracle.reply(imp, -(-F // alpha), P, n, q, b, N, m)
        assert np.array_equal(ctx.reply(d, n, q), want)


def undecided(q: np.ndarray, n, N, m, moduli, kind: str) -> np.ndarray:
    """The query with words that the sums must refuse or survive."""
    w = q.reshape(sum(n), 2, m, N).copy()
    p = moduli[0]
    if kind == "one word p":
        w[n[0] // 2, 1, 0, 3] = p
    elif kind == "unreduced last word":
        w[-1, 0, m - 1, N - 1] = 2**64 - 1
    elif kind == "zero words":
        w[:, :, :, ::2] = 0
    elif kind == "zero query":
        w[:] = 0
    elif kind == "constant words":
        w[:] = w[0]
    elif kind == "arbitrary words":
        return random_query(77, n, N, m, moduli, reduced=False)
    return w.reshape(-1)


@pytest.mark.parametrize("kind", ["one word p", "unreduced last word", "zero words", "zero query", "constant words",
                                  "arbitrary words"])
@pytest.mark.parametrize("N,m,n,F,L", [(512, 2, [450], 450, 500), (1024, 1, [70, 30], 600, 300)])
def test_words_sums_cannot_decide(engine, oracle, N, m, n, F, L, kind):
    b, P = shapes(N, m, n, 1, L, oracle)
    q = undecided(random_query(41, n, N, m, oracle.moduli(m)), n, N, m, oracle.moduli(m), kind)
    elems = random_db(42, F, L)
    if kind == "constant words":
        elems = np.tile(elems[:L], F)  # equal elements too: the same term in every slot
    with engine.Context(N, m) as ctx:
        d = ctx.import_db(elems, F, L, 1, b)
        want = oracle.reply(d.export(), F, P, n, q, b, N, m)
        assert np.array_equal(ctx.reply(d, n, q), want)
        ordinary = random_query(43, n, N, m, oracle.moduli(m))
        assert np.array_equal(ctx.reply(d, n, ordinary), oracle.reply(d.export(), F, P, n, ordinary, b, N, m))


@pytest.mark.parametrize("zeros", [slice(0, None), slice(200, 300), slice(430, None), slice(0, None, 2)])
def test_elements_of_zero_bytes(engine, oracle, zeros):
    """All-zero elements import to words 0 and p, whose terms keep chains apart."""
    N, m, n, F, L = 1024, 2, [450], 450, 1500
    b, P = shapes(N, m, n, 1, L, oracle)
    elems = random_db(51, F, L).reshape(F, L)
    elems[zeros] = 0
    q = random_query(52, n, N, m, oracle.moduli(m))
    with engine.Context(N, m) as ctx:
        d = ctx.import_db(elems.reshape(-1), F, L, 1, b)
        assert np.array_equal(ctx.reply(d, n, q), oracle.reply(d.export(), F, P, n, q, b, N, m))


@pytest.mark.parametrize("use_graph", [False, True])
def test_batches_of_sums(engine, oracle, use_graph):
    """Batched and captured: several queries per launch (runs with a finish kernel, one run
    per column, idle groups), one of them with an unreduced word, replayed with other words."""
    torch = pytest.importorskip("torch")
    N, m = 1024, 2
    with engine.Context(N, m) as ctx:
        items, want = [], []
        for k, (n, alpha, F, L) in enumerate([([500], 1, 500, 800), ([100, 40], 1, 3950, 300), ([70, 60], 2, 500, 500)]):
            b, P = shapes(N, m, n, alpha, L, oracle)
            d = ctx.import_db(random_db(60 + k, F, L), F, L, alpha, b)
            imp = d.export()
            for s in range(2):
                out = None
                per = []
                for version in range(2):
                    q = random_query(600 + 10 * k + 2 * s + version, n, N, m, oracle.moduli(m))
                    if version and k == 1:
                        q[12345] = 2**63 + 5
                    per.append((q, oracle.reply(imp, -(-F // alpha), P, n, q, b, N, m)))
                out = torch.full((per[0][1].size,), -1, dtype=torch.int64, device="cuda")
                qd = torch.empty(per[0][0].size, dtype=torch.int64, device="cuda")
                items.append((d, n, qd, out))
                want.append(per)
        for version in (0, 1, 0):
            for (_, _, qd, out), per in zip(items, want):
                qd.copy_(torch.from_numpy(per[version][0].view(np.int64)))
                out.fill_(-1)
            torch.cuda.synchronize()
            ctx.reply_batch(items, use_graph=use_graph)
            for (_, _, _, out), per in zip(items, want):
                assert np.array_equal(out.cpu().numpy().view(np.uint64), per[version][1])


@pytest.mark.parametrize("n,alpha,F", [([500], 1, 500), ([70, 60], 2, 500), ([6, 10, 9], 1, 150)])
def test_noalloc_takes_the_same_levels(engine, oracle, n, alpha, F):
    torch = pytest.importorskip("torch")
    N, m, L = 1024, 1, 500
    b, P = shapes(N, m, n, alpha, L, oracle)
    fn = engine.lib().xpir_b200_reply_noalloc
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint32, ctypes.POINTER(ctypes.c_uint32),
                   ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint64, ctypes.POINTER(ctypes.c_uint64)]
    with engine.Context(N, m) as ctx:
        d = ctx.import_db(random_db(71, F, L), F, L, alpha, b)
        for bad in (False, True):
            q = random_query(72 + bad, n, N, m, oracle.moduli(m))
            if bad:
                q[-5] = 2**62
            want = oracle.reply(d.export(), -(-F // alpha), P, n, q, b, N, m)
            qd = torch.from_numpy(q.view(np.int64)).cuda()
            out = torch.full((want.size,), -1, dtype=torch.int64, device="cuda")
            cnt = ctypes.c_uint64()
            assert fn(ctx.handle, d.handle, len(n), (ctypes.c_uint32 * len(n))(*n), qd.data_ptr(), out.data_ptr(),
                      out.numel() * 8, ctypes.byref(cnt)) == engine.OK
            assert np.array_equal(out.cpu().numpy().view(np.uint64), want)
