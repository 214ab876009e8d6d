"""Extraction of many ciphertexts (one CTA each decrypts, lifts and packs) against the oracle:
one to four moduli (one- and two-word values), two levels, element sizes that end inside a
word, odd output addresses, reduced and arbitrary words.  Bytes: no tolerance."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,m,n,polys,cut,reduced", [
    (512, 1, [20], 300, 0, True), (512, 2, [20], 296, 3, True), (1024, 3, [8], 301, 5, True),
    (512, 4, [9], 297, 1, False), (2048, 2, [50], 299, 7, True), (512, 2, [6, 5], 120, 2, True),
    (4096, 3, [5], 296, 0, True)])
def test_many_ciphertexts_match_oracle(engine, oracle, N, m, n, polys, cut, reduced):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(N + m)
    d, b = len(n), oracle.bits_per_coeff(N, m, n[0])
    L = polys * (b * N // 8) - cut
    key = np.concatenate([rng.integers(0, p, size=N, dtype=np.uint64) for p in oracle.moduli(m)])
    nct = oracle.extract_count(L, d, b, N, m)
    assert nct >= 296  # enough for a CTA per ciphertext (at level 2, then at level 1 too or not)
    ct = rng.integers(0, 2**64, size=(nct, 2, m, N), dtype=np.uint64)
    if reduced:
        for c, p in enumerate(oracle.moduli(m)):
            ct[:, :, c, :] %= np.uint64(p)
    ct = ct.reshape(-1)
    want = oracle.extract(ct, key, d, b, N, m, L)
    with engine.Context(N, m) as ctx:
        assert np.array_equal(ctx.extract(key, d, b, L, ct), want)
        dct = torch.from_numpy(ct.view(np.int64)).cuda()
        for shift in (0, 3):
            buf = torch.full((L + 16,), 0xA5, dtype=torch.uint8, device="cuda")
            ctx.extract(key, d, b, L, dct, buf[shift:shift + L])
            got = buf.cpu().numpy()
            assert np.array_equal(got[shift:shift + L], want)
            assert (got[:shift] == 0xA5).all() and (got[shift + L:] == 0xA5).all()
