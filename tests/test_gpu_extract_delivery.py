"""Where extraction leaves the element: lengths that the float arithmetic of the ciphertext
count falls short of (the bytes past the last ciphertext's plaintext are zero, whatever the
caller's buffer held), and buffers that overlap the replies.  Bytes: no tolerance."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def random_words(seed, oracle, N, m, *shape):
    w = np.random.default_rng(seed).integers(0, 2**64, size=(*shape, m, N), dtype=np.uint64)
    for c, p in enumerate(oracle.moduli(m)):
        w[..., c, :] %= np.uint64(p)
    return w.reshape(-1)


# 1500 and 1599 ciphertexts take a CTA each, 130 the two kernels; one byte more than they hold.
@pytest.mark.parametrize("N,m,b,polys", [(2048, 2, 46, 1500), (2048, 2, 41, 1599), (8192, 3, 127, 130)])
def test_bytes_past_the_last_ciphertext_are_zero(engine, oracle, N, m, b, polys):
    torch = pytest.importorskip("torch")
    held = polys * (b * N // 8)
    L = held + 1
    assert engine.extract_count(L, 1, b, N, m) == polys
    key, ct = random_words(5, oracle, N, m), random_words(6, oracle, N, m, polys, 2)
    want = np.concatenate([oracle.extract(ct, key, 1, b, N, m, held), np.zeros(1, dtype=np.uint8)])
    with engine.Context(N, m) as ctx:
        assert np.array_equal(ctx.extract(key, 1, b, L, ct), want)
        dct = torch.from_numpy(ct.view(np.int64)).cuda()
        for shift in (0, 8, 3):
            buf = torch.full((L + 24,), 0xA5, dtype=torch.uint8, device="cuda")
            ctx.extract(key, 1, b, L, dct, buf[shift:shift + L])
            got = buf.cpu().numpy()
            assert np.array_equal(got[shift:shift + L], want)
            assert (got[:shift] == 0xA5).all() and (got[shift + L:] == 0xA5).all()


def test_many_bytes_past_the_last_ciphertext(engine, oracle):
    """A long element that the count falls 31 bytes short of, more than three words."""
    torch = pytest.importorskip("torch")
    N, m, b, polys, over = 512, 1, 17, 560000, 31
    held = polys * (b * N // 8)
    assert engine.extract_count(held + over, 1, b, N, m) == polys == engine.extract_count(held, 1, b, N, m)
    p = oracle.moduli(m)[0]
    gen = torch.Generator(device="cuda").manual_seed(7)
    ct = torch.randint(0, p, (polys * 2 * N,), dtype=torch.int64, device="cuda", generator=gen)
    key = random_words(8, oracle, N, m)
    with engine.Context(N, m) as ctx:
        short = torch.full((held,), 0xA5, dtype=torch.uint8, device="cuda")
        ctx.extract(key, 1, b, held, ct, short)
        few = 40  # the first ciphertexts against the oracle, all of them against the exact length
        want = oracle.extract(ct[:few * 2 * N].cpu().numpy().view(np.uint64), key, 1, b, N, m, few * (b * N // 8))
        assert np.array_equal(short[:want.size].cpu().numpy(), want)
        for shift in (0, 3):
            buf = torch.full((held + over + 16,), 0xA5, dtype=torch.uint8, device="cuda")
            ctx.extract(key, 1, b, held + over, ct, buf[shift:shift + held + over])
            assert torch.equal(buf[shift:shift + held], short)
            assert (buf[shift + held:shift + held + over] == 0).all()
            assert (buf[:shift] == 0xA5).all() and (buf[shift + held + over:] == 0xA5).all()
        host = np.full(held + over, 0xA5, dtype=np.uint8)
        ctx.extract(key, 1, b, held + over, ct, host)
        assert np.array_equal(host[:held], short.cpu().numpy()) and not host[held:].any()


@pytest.mark.parametrize("N,m,polys", [(2048, 2, 900), (512, 1, 3000)])
@pytest.mark.parametrize("at", ["start", "middle", "last words"])
def test_in_place(engine, oracle, N, m, polys, at):
    """The element over the replies it comes from: every ciphertext is read before any byte
    is written."""
    torch = pytest.importorskip("torch")
    b = oracle.bits_per_coeff(N, m, 20)
    L = polys * (b * N // 8)
    assert engine.extract_count(L, 1, b, N, m) == polys
    key, ct = random_words(15, oracle, N, m), random_words(16, oracle, N, m, polys, 2)
    want = oracle.extract(ct, key, 1, b, N, m, L)
    first = {"start": 0, "middle": ct.nbytes // 2, "last words": ct.nbytes - 8}[at]
    with engine.Context(N, m) as ctx:
        buf = torch.full((ct.nbytes + L,), 0xA5, dtype=torch.uint8, device="cuda")
        buf[:ct.nbytes] = torch.from_numpy(ct.view(np.uint8)).cuda()
        torch.cuda.synchronize()
        ctx.extract(key, 1, b, L, buf[:ct.nbytes], buf[first:first + L])
        got = buf.cpu().numpy()
        assert np.array_equal(got[first:first + L], want)
        assert np.array_equal(got[:first], ct.view(np.uint8)[:first])
        assert np.array_equal(got[first + L:ct.nbytes], ct.view(np.uint8)[first + L:])
        assert (got[max(first + L, ct.nbytes):] == 0xA5).all()
