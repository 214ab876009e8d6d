"""Generated queries in device buffers that start off a 16-byte boundary (the kernel stores
pairs of words): the same words, and nothing written beside them."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_query_at_any_word(engine, oracle, shift):
    torch = pytest.importorskip("torch")
    N, m, n, chosen = 1024, 2, [5, 4], 13
    key = oracle.seeded_prng_key(3)
    sk = oracle.keygen(key, 0, N, m)
    b = oracle.bits_per_coeff(N, m, n[0])
    want = oracle.query(key, 1, sk, n, chosen, b, N, m)
    with engine.Context(N, m) as ctx:
        buf = torch.full((want.size + 4,), -1, dtype=torch.int64, device="cuda")
        ctx.generate_query(key, 1, sk, n, chosen, b, out=buf[shift:shift + want.size])
        got = buf.cpu().numpy()
    assert np.array_equal(got[shift:shift + want.size].view(np.uint64), want)
    assert (got[:shift] == -1).all() and (got[shift + want.size:] == -1).all()
