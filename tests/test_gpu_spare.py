"""The memory of a freed database serves the context's next import: imports of other sizes
after a free hold the oracle's words, two live databases never share memory, and closing the
context gives the block back."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import random_db

pytestmark = pytest.mark.gpu


def test_imports_after_frees(engine, oracle):
    torch = pytest.importorskip("torch")
    N, m, L = 1024, 2, 1000
    b = oracle.bits_per_coeff(N, m, 40)
    torch.cuda.synchronize()
    with engine.Context(N, m) as ctx:
        live = []
        for k, F in enumerate((40, 39, 25, 12, 60, 60, 3)):
            elems = random_db(80 + k, F, L)
            db = ctx.import_db(elems, F, L, 1, b)
            live.append((db, oracle.import_db(elems, F, L, 1, b, N, m)))
            for d, want in live:
                assert np.array_equal(d.export(), want)
            if k != 3:  # one stays alive
                live.pop()[0].free()
    with engine.Context(N, m) as ctx:
        F = 20000  # 328 MB of words, kept after the free
        elems = torch.zeros(F * 64, dtype=torch.uint8, device="cuda")
        ctx.import_db(elems, F, 64, 1, b).free()
        ctx.synchronize()
        held = torch.cuda.mem_get_info()[0]
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] - held >= F * m * N * 8
