"""Replies written over a query they come from.  A query word not below its modulus makes
the engine repeat a reply, which reads the query a second time: the replies must not have
replaced it by then.  Integer work: bit-exact, no tolerance."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from helpers import random_db, random_query, shapes

pytestmark = pytest.mark.gpu

# Level 1's ciphertexts are read before the last level writes a reply, and one run of a lone
# column reads a coefficient's whole column before it writes it: the replies may lie there.
N, M = 1024, 1
CASES = [([100, 64], 1, 6400, 200), ([700], 1, 700, 1500)]  # level 1 by residue sums


def make(oracle, n, alpha, F, L, seed, bad):
    b, P = shapes(N, M, n, alpha, L, oracle)
    q = random_query(seed, n, N, M, oracle.moduli(M))
    if bad:
        q[(n[0] - 1) * 2 * M * N + 5] = 2**62  # in level 1's last ciphertext
    return b, P, q


@pytest.mark.parametrize("bad", [False, True])
@pytest.mark.parametrize("call", ["reply", "noalloc", "batch", "graph"])
@pytest.mark.parametrize("n,alpha,F,L", CASES)
def test_replies_over_their_query(engine, oracle, n, alpha, F, L, call, bad):
    torch = pytest.importorskip("torch")
    b, P, q = make(oracle, n, alpha, F, L, 91, bad)
    with engine.Context(N, M) as ctx:
        d = ctx.import_db(random_db(90, F, L), F, L, alpha, b)
        want = oracle.reply(d.export(), -(-F // alpha), P, n, q, b, N, M)
        for _ in range(2):
            buf = torch.from_numpy(q.view(np.int64)).cuda()
            out = buf[:want.size]
            torch.cuda.synchronize()
            if call == "reply":
                ctx.reply(d, n, buf, out)
            elif call == "noalloc":
                fn = engine.lib().xpir_b200_reply_noalloc
                fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint32, ctypes.POINTER(ctypes.c_uint32),
                               ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint64, ctypes.POINTER(ctypes.c_uint64)]
                assert fn(ctx.handle, d.handle, len(n), (ctypes.c_uint32 * len(n))(*n), buf.data_ptr(),
                          out.data_ptr(), want.nbytes, ctypes.byref(ctypes.c_uint64())) == engine.OK
            else:
                ctx.reply_batch([(d, n, buf, out)], use_graph=call == "graph")
            assert np.array_equal(out.cpu().numpy().view(np.uint64), want)


@pytest.mark.parametrize("use_graph", [False, True])
def test_replies_over_an_earlier_query_of_the_batch(engine, oracle, use_graph):
    """Queries of one database and grid are replied to before those of the next: a later
    one's replies may lie over an earlier query."""
    torch = pytest.importorskip("torch")
    n, alpha, F, L = [700], 1, 700, 1500
    with engine.Context(N, M) as ctx:
        items, want, bufs = [], [], []
        for k, bad in enumerate((True, False)):
            b, P, q = make(oracle, n, alpha, F, L, 93 + k, bad)
            d = ctx.import_db(random_db(92 + k, F, L), F, L, alpha, b)
            want.append(oracle.reply(d.export(), F, P, n, q, b, N, M))
            bufs.append(torch.from_numpy(q.view(np.int64)).cuda())
            items.append([d, n, bufs[k], torch.full((want[k].size,), -1, dtype=torch.int64, device="cuda")])
        items[1][3] = bufs[0][4096:4096 + want[1].size]
        torch.cuda.synchronize()
        ctx.reply_batch([tuple(i) for i in items], use_graph=use_graph)
        for item, w in zip(items, want):
            assert np.array_equal(item[3].cpu().numpy().view(np.uint64), w)
