"""The residue-sum kernel's bounded waits, made to run out on purpose
(xpir_b200_ctx_set_wait_test), as test_gpu_wait_timeout.py does for either kernel: levels cut
into runs with a finish kernel, and one run per column with one to four columns a CTA.  The
producer issues no copy that it does not wait for and every wait is bounded, so the CTAs
return with nothing in flight; the context then answers the next query bit-exactly."""
from __future__ import annotations

import time

import numpy as np
import pytest

from helpers import random_db, random_query, shapes

pytestmark = pytest.mark.gpu

SHORT_LIMIT = 4096  # polls per wait; each poll suspends for at most 20 us


# N, m, grid, elements, bytes, launches of a reply
@pytest.mark.parametrize("N,m,n,F,L,count", [
    (2048, 2, [3000], 3000, 4096, 2),   # one column, runs
    (1024, 1, [1000], 1000, 14000, 2),  # eight columns, runs
    (512, 1, [700], 700, 2500, 2),      # three columns, runs
    (512, 2, [30, 130], 3900, 60, 3),   # two columns a CTA, one run, then a short level by slot
    (512, 2, [133, 300], 39870, 60, 3)])  # four columns a CTA, a level of 300 slots after it
def test_withheld_tile_of_the_sums(engine, oracle, N, m, n, F, L, count):
    b, P = shapes(N, m, n, 1, L, oracle)
    q = random_query(141, n, N, m, oracle.moduli(m))
    with engine.Context(N, m) as ctx:
        d = ctx.import_db(random_db(140, F, L), F, L, 1, b)
        want = oracle.reply(d.export(), F, P, n, q, b, N, m)

        def launches():
            before = ctx.launch_count
            assert np.array_equal(ctx.reply(d, n, q), want)
            return ctx.launch_count - before

        usual = launches()
        ctx.set_wait_test(SHORT_LIMIT, -1)
        assert launches() == usual  # a short limit alone changes neither route nor reply
        ctx.set_wait_test(SHORT_LIMIT, 1)
        before, t0 = ctx.launch_count, time.perf_counter()
        with pytest.raises(engine.XpirError) as err:
            ctx.reply(d, n, q)
        assert err.value.status == engine.ERR_TIMEOUT
        assert time.perf_counter() - t0 < 60
        assert ctx.launch_count - before >= usual
        ctx.set_wait_test(0, -1)
        assert launches() == usual == count
