"""Performance cases of the engine, through the Python binding a user's program calls.

Each case is one call of the server or of the client on one GPU: a reply to a query (small,
ordinary and large databases, one to three recursion levels, query in device or in host
memory), a batch of queries, the import of a database together with the first reply from
it, the generation of a query, and the extraction of an element from replies.  The sizes
are the benchmark's configurations and sizes of the tests' ranges.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what the program holds before the call (context, database, query)
    run(state)           one call, its outputs whole
    work(case)           bytes and operations that the call cannot do without
    exact(case, seed)    None: every output is a modular integer or a byte (see below)
"""
from __future__ import annotations

import numpy as np
import torch

import xpir_b200 as xb


def _case(name, op, N, m, n, F=0, L=0, alpha=1, host=False, queries=1):
    n = list(n) + [0] * (3 - len(n))
    return {"name": name, "op": op, "N": N, "m": m, "n0": n[0], "n1": n[1], "n2": n[2], "F": F, "L": L,
            "alpha": alpha, "host": host, "queries": queries}


def listed() -> list[dict]:
    return [
        # The smallest call: a query on a directory of a hundred short records.
        _case("reply_tiny", "reply", 1024, 1, [100], 100, 900),
        # The plain single query: 1,000 files of 12 KB, one modulus.
        _case("reply_plain", "reply", 1024, 1, [1000], 1000, 12288),
        # The large flat database: 100,000 x 4 KB, where query and database cross HBM once.
        _case("reply_flat_large", "reply", 2048, 2, [100000], 100000, 4096),
        # The large recursive database: 1,048,576 x 256 B, 16 to an element, on a 1024 x 1024 grid.
        _case("reply_recursive_large", "reply", 4096, 3, [1024, 1024], 1048576, 256, 16),
        # Ragged sizes: a prime number of odd-sized elements, three to a group, a short last
        # group and a grid larger than the database.
        _case("reply_ragged", "reply", 2048, 2, [61, 55], 9973, 5003, 3),
        # Three recursion levels on a small grid.
        _case("reply_three_levels", "reply", 2048, 2, [30, 20, 12], 7001, 1500),
        # A server's call: the query arrives in pinned host memory, the reply goes back to the host.
        _case("reply_host_query", "reply", 2048, 2, [256, 256], 65536, 8192, host=True),
        # Eight queries of three shapes on one database, submitted together.
        _case("batch_mixed", "batch", 2048, 2, [256, 256], 65536, 8192, queries=8),
        # A new database: import of device-resident elements and the first reply from it.
        _case("import_and_reply", "import", 2048, 2, [142, 141], 20000, 4096),
        # The client's query for the large recursive grid.
        _case("query_generation", "query", 4096, 3, [1024, 1024]),
        # The client's side of one 50 MB element.
        _case("extract_large", "extract", 2048, 2, [100000], L=50_000_000),
        # The client's side of one recursive reply, in host memory.
        _case("extract_two_levels", "extract", 2048, 2, [256, 256], L=8192, host=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng) -> dict:
    op = rng.choice(["reply", "reply", "reply", "reply", "batch", "import", "query", "extract"])
    N, m = rng.choice([(1024, 1), (1024, 2), (2048, 2), (2048, 2), (4096, 2), (4096, 3)])
    ct = 16 * m * N  # bytes of a ciphertext
    alpha = rng.choice([1, 1, 1, 2, 3, 4, 16])
    if op == "query":
        count = _log_int(rng, 60, min(6000, 400_000_000 // ct))
        n = [count] if rng.random() < 0.5 else [count // 2 + 1, count - count // 2]
        return _case("", op, N, m, n)
    if op == "extract":
        d = rng.choice([1, 1, 2])
        n = [_log_int(rng, 50, 50000)] if d == 1 else [_log_int(rng, 8, 400), _log_int(rng, 8, 400)]
        return _case("", op, N, m, n, L=_log_int(rng, 700, 40_000_000 if d == 1 else 60_000), host=rng.random() < 0.3)
    # database of at most 2 GB of elements' polys, query of at most 2.5 GB
    L = _log_int(rng, 250, 20000)
    b = 46 if m == 2 else (16 if m == 1 else 74)
    groups_max = int(2e9 / (8 * m * N * max(1, -(-8 * alpha * L // (b * N)))))
    groups = _log_int(rng, 60, max(61, min(groups_max, 150_000)))
    F = max(1, groups * alpha - rng.randrange(alpha))
    d = rng.choice([1, 2, 2, 3])
    if d == 1 and groups * ct > 2_500_000_000:
        d = 2
    if d == 1:
        n = [groups]
    elif d == 2:
        n0 = max(2, int(groups**0.5 * (0.7 + 0.6 * rng.random())))
        n = [n0, -(-groups // n0) + rng.randrange(3)]
    else:
        n0 = max(2, int(groups ** (1 / 3) * (0.8 + 0.5 * rng.random())))
        n1 = max(2, int(groups ** (1 / 3) * (0.8 + 0.4 * rng.random())))
        n = [n0, n1, -(-groups // (n0 * n1)) + rng.randrange(2)]
    if op == "batch":
        return _case("", op, N, m, n, F, L, alpha, queries=rng.choice([2, 3, 4, 8]) if d > 1 else 2)
    return _case("", op, N, m, n, F, L, alpha, host=(op == "reply" and rng.random() < 0.2))


def _levels(case) -> list[int]:
    return [case[k] for k in ("n0", "n1", "n2") if case[k]]


def _batch_shapes(case) -> list[tuple[list[int], int]]:
    """(grid, alpha) of a batch's queries: mostly the case's grid; with four queries or more
    a quarter of them one-level and a quarter one-level with four times the aggregation."""
    n, a, k = _levels(case), case["alpha"], case["queries"]
    flat = -(-case["F"] // a), -(-case["F"] // (4 * a))
    few = k // 4 if k >= 4 and flat[0] * 16 * case["m"] * case["N"] <= 4_500_000_000 else 0
    return [([flat[0]], a)] * few + [([flat[1]], 4 * a)] * few + [(n, a)] * (k - 2 * few)


def _words(N, m, count, halves, gen) -> torch.Tensor:
    """`count` ciphertexts (or keys) of uniform residues, [count][halves][m][N]."""
    t = torch.empty((count, halves, m, N), dtype=torch.int64, device="cuda")
    step = max(1, (1 << 27) // (halves * m * N))
    for c, p in enumerate(xb.moduli(m)):
        for i in range(0, count, step):
            k = min(step, count - i)
            t[i:i + k, :, c] = torch.randint(0, p, (k, halves, N), dtype=torch.int64, device="cuda", generator=gen)
    return t.reshape(-1)


def _reply_words(ctx, db, n) -> int:
    P = db.polys_per_element
    for _ in n[1:]:
        P = xb.polys_per_element(P * ctx.ct_words * 8, 1, db.bits_per_coeff, ctx.N)
    return P * ctx.ct_words


def _pinned(t: torch.Tensor) -> np.ndarray:
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy().view(np.uint64)


def prepare(case, seed) -> dict:
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    N, m, n, op = case["N"], case["m"], _levels(case), case["op"]
    ctx = xb.Context(N, m)
    st = {"op": op, "ctx": ctx, "n": n, "b": xb.bits_per_coeff(N, m, n[0]), "case": case}
    if op in ("query", "extract"):
        st["sk"] = _words(N, m, 1, 1, gen).cpu().numpy().view(np.uint64)
    if op == "query":
        st["key"] = np.random.default_rng(seed).integers(0, 256, size=32, dtype=np.uint8)
        st["chosen"] = int(np.random.default_rng(seed + 1).integers(0, int(np.prod(n))))
        st["out"] = torch.empty(sum(n) * ctx.ct_words, dtype=torch.int64, device="cuda")
    elif op == "extract":
        count = xb.extract_count(case["L"], len(n), st["b"], N, m)
        replies = _words(N, m, count, 2, gen)
        if case["host"]:
            st["replies"], st["out"] = _pinned(replies), np.zeros(case["L"], dtype=np.uint8)
        else:
            st["replies"], st["out"] = replies, torch.empty(case["L"], dtype=torch.uint8, device="cuda")
    else:
        elems = torch.randint(0, 256, (case["F"] * case["L"],), dtype=torch.uint8, device="cuda", generator=gen)
        if op == "batch":
            st["items"], dbs = [], {}
            for grid, alpha in _batch_shapes(case):
                key = (alpha, xb.bits_per_coeff(N, m, grid[0]))
                if key not in dbs:
                    dbs[key] = ctx.import_db(elems, case["F"], case["L"], alpha, key[1])
                q = _words(N, m, sum(grid), 2, gen)
                out = torch.empty(_reply_words(ctx, dbs[key], grid), dtype=torch.int64, device="cuda")
                st["items"].append((dbs[key], grid, q, out))
        else:
            q = _words(N, m, sum(n), 2, gen)
            st["query"] = _pinned(q) if case["host"] else q
            if op == "import":
                st["elems"] = elems
            else:
                st["db"] = ctx.import_db(elems, case["F"], case["L"], case["alpha"], st["b"])
                words = _reply_words(ctx, st["db"], n)
                st["out"] = (np.empty(words, dtype=np.uint64) if case["host"]
                             else torch.empty(words, dtype=torch.int64, device="cuda"))
        ctx.synchronize()
    torch.cuda.synchronize()
    return st


def run(st):
    ctx, op, case = st["ctx"], st["op"], st["case"]
    if op == "reply":
        return ctx.reply(st["db"], st["n"], st["query"], st["out"])
    if op == "batch":
        ctx.reply_batch(st["items"])
        return [out for *_, out in st["items"]]
    if op == "import":
        db = ctx.import_db(st["elems"], case["F"], case["L"], case["alpha"], st["b"])
        out = torch.empty(_reply_words(ctx, db, st["n"]), dtype=torch.int64, device="cuda")
        ctx.reply(db, st["n"], st["query"], out)
        db.free()
        return out
    if op == "query":
        return ctx.generate_query(st["key"], 1, st["sk"], st["n"], st["chosen"], st["b"], out=st["out"])
    return ctx.extract(st["sk"], len(st["n"]), st["b"], case["L"], st["replies"], st["out"])


def _reply_work(N, m, n, F, L, alpha) -> tuple[int, int]:
    """Bytes (imported database, query, replies once each) and operations (a multiplication
    and an addition per database word and ciphertext half, at every level)."""
    b = xb.bits_per_coeff(N, m, n[0])
    P, real, words = xb.polys_per_element(L, alpha, b, N), -(-F // alpha), 0
    total = sum(n) * 16 * m * N
    for lvl, n_i in enumerate(n):
        words += real * P * m * N
        if lvl == 0:
            total += words * 8
        real = -(-real // n_i)
        if lvl + 1 < len(n):
            P = xb.polys_per_element(P * 16 * m * N, 1, b, N)
    return total + P * 16 * m * N, 4 * words


def work(case) -> dict:
    N, m, n, op = case["N"], case["m"], _levels(case), case["op"]
    b, logn = xb.bits_per_coeff(N, m, n[0]), N.bit_length() - 1
    transform = N // 2 * logn + N  # modular products of one twisted transform
    if op in ("reply", "import"):
        nbytes, ops = _reply_work(N, m, n, case["F"], case["L"], case["alpha"])
        if op == "import":  # the imported words are written once as well
            groups = -(-case["F"] // case["alpha"])
            polys = groups * xb.polys_per_element(case["L"], case["alpha"], b, N) * m
            nbytes += case["F"] * case["L"] + polys * N * 8
            ops += polys * transform * 2
        return {"bytes": nbytes, "flops": ops}
    if op == "batch":
        nbytes = ops = 0
        seen = set()
        for grid, alpha in _batch_shapes(case):
            nb, o = _reply_work(N, m, grid, case["F"], case["L"], alpha)
            bb = xb.bits_per_coeff(N, m, grid[0])
            if (alpha, bb) in seen:  # a database crosses once for all its queries
                nb -= -(-case["F"] // alpha) * xb.polys_per_element(case["L"], alpha, bb, N) * m * N * 8
            seen.add((alpha, bb))
            nbytes, ops = nbytes + nb, ops + o
        return {"bytes": nbytes, "flops": ops}
    if op == "query":
        polys = sum(n) * m
        return {"bytes": polys * 16 * N, "flops": polys * (transform + 2 * N) * 2}
    count = xb.extract_count(case["L"], len(n), b, N, m)
    return {"bytes": count * 16 * m * N + case["L"], "flops": count * m * (transform + 2 * N) * 2}


def exact(case, seed):
    """Replies, queries and elements are modular words and bytes, not approximations of real
    numbers: they have one right value each and are compared for equality."""
    return None
