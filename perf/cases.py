"""The calls whose speed this repository cares about, as cases that can be prepared, run and checked.

Each case is one call (or one short program) on the public surface of ``clwilson_b200``.  The ranges of test
primes are placed by the seed inside the case's neighbourhood, so that every seed gives other primes, class
targets and exponents.  The kinds:

  search   ``Engine.search``: a full search of one range, result lines and checksum (the command line's job)
  rows     ``Engine.rows``: every test prime's digits; with ``q_cap`` the capped column product that the
           mid-size and top-of-range configurations measure
  batch    ``Engine.batch``: many ranges, log-uniform starts and widths, one call
  serve    ``Server``: a burst of range requests against a resident session, until every one is done
  pieces   ``Engine.rows_from`` + ``Engine.search_from``: a search cut at a column, as checkpoints cut it
  product  ``Engine.rows_product``: the row-wise product of the column pieces of several GPUs
  noalloc  ``wl_column_product_noalloc`` on device arrays of the caller's

Integers come back as int64 arrays of the same bits, padded with zeros to a length that the case alone sets (a range of
another seed holds a few more or fewer primes).
"""
import ctypes
import math
import random

import numpy as np
import torch

import clwilson_b200 as wl

TOP = 2 ** 62 - 1


def listed():
    return [
        # the reference's self-test size: nothing but launches, copies and host work
        {"name": "search-tiny", "kind": "search", "pmin": 200, "width": 364, "fresh": False},
        # a quick range of small primes, every row read back
        {"name": "rows-1e7", "kind": "rows", "pmin": 10 ** 7, "width": 20011, "q_cap": 0},
        # the headline configuration: 1e6 integers from 1e9, columns sieved in the call as every run of the
        # command line does
        {"name": "search-1e9", "kind": "search", "pmin": 10 ** 9, "width": 10 ** 6, "fresh": True},
        # a short work unit of the same size of primes on a resident engine
        {"name": "search-1e9-narrow", "kind": "search", "pmin": 10 ** 9, "width": 20000, "fresh": False},
        # a short full search whose columns pass 2^32: the windowed sieve and its sweep
        {"name": "search-past-2^32", "kind": "search", "pmin": 2 * 10 ** 10, "width": 501, "fresh": False},
        # the mid-size configuration (3 limbs), capped
        {"name": "rows-mid", "kind": "rows", "pmin": 10 ** 13, "width": 100000, "q_cap": 2 ** 29 + 1235},
        # the top of the range (4 limbs), capped: exponents change at every column
        {"name": "rows-top", "kind": "rows", "pmin": TOP - 2 * 10 ** 6, "width": 50000, "q_cap": 2 ** 27},
        # many ranges in one call, sizes over two orders of magnitude
        {"name": "batch-64", "kind": "batch", "ranges": 64, "width": 20000, "q_cap": 2 ** 24},
        # a burst of small requests at a serving session
        {"name": "serve-64", "kind": "serve", "ranges": 64, "width": 2000, "q_cap": 2 ** 24},
        # checkpoint and resume: a capped piece, then the finish from its products
        {"name": "pieces-1e8", "kind": "pieces", "pmin": 10 ** 8, "width": 200001, "cut": 2 ** 22},
        # folding the pieces of eight GPUs
        {"name": "product-8", "kind": "product", "rows": 48155, "parts": 8, "bits": 30},
        # the column product for hosts that own all device memory
        {"name": "noalloc-2000", "kind": "noalloc", "rows": 2000, "bits": 30, "q_cap": 2 ** 24},
    ]


# ---------------------------------------------------------------------------
# sizes
# ---------------------------------------------------------------------------

def _pi(x):
    """About how many primes are below x."""
    return 0.0 if x < 2 else x / max(1.0, math.log(x) - 1.0) if x > 60 else x / 2.5


def _rows(pmin, width):
    return max(1.0, width / math.log(pmin + width))


def _cells(pmin, width, q_cap=0):
    """Row x column products of one range: half its primes go to (p-1)/6, a quarter each to /4 and /2."""
    n = _rows(pmin, width)
    cut = (lambda t: min(t, q_cap)) if q_cap else (lambda t: t)
    return n * (0.5 * _pi(cut(pmin / 6)) + 0.25 * _pi(cut(pmin / 4)) + 0.25 * _pi(cut(pmin / 2)))


def _ranges(case, seed):
    """Log-uniform starts in [1e8, 2^62 - 1e7) from the seed and log-uniform widths up to the case's, as the
    batched and serving configurations draw them."""
    r, rw = random.Random(seed * 7919 + 17), random.Random(case["ranges"])
    out = []
    for _ in range(case["ranges"]):
        a = int(math.exp(r.uniform(math.log(1e8), math.log(2.0 ** 62 - 1e7))))
        w = int(math.exp(rw.uniform(math.log(max(300.0, case["width"] / 50)), math.log(case["width"]))))
        out.append((a, min(a + w, TOP)))
    return out


def _place(case, seed):
    """The case's range, moved by the seed by up to 1% of its start (at least 1,000)."""
    r = random.Random(seed * 104729 + 5)
    a = case["pmin"]
    off = r.randrange(0, max(1000, min(a // 100, 10 ** 9)))
    if a + off + case["width"] > TOP:
        off = r.randrange(0, TOP - case["width"] - a)
    return a + off, a + off + case["width"]


def _cost(c):
    """Column products of a case, those where the exponent changes at every column counted with what
    raising to it takes."""
    if c["kind"] in ("search", "pieces"):
        return _cells(c["pmin"], c["width"]) + 3e9 * (c["pmin"] > 8.5e9) * c["pmin"] / 2e10
    if c["kind"] == "rows":
        return _cells(c["pmin"], c["width"], c["q_cap"]) * (8 if c["q_cap"] and c["q_cap"] ** 2 < c["pmin"] else 1)
    if c["kind"] in ("batch", "serve"):
        return c["ranges"] * 0.5 * c["width"] / 32 * _pi(c["q_cap"]) * 8
    if c["kind"] == "product":
        return c["rows"] * c["parts"] * 1e3
    return c["rows"] * _pi(c["q_cap"])


def draw(rng):
    def log(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    while True:
        k = rng.choice(["search", "search", "past", "rows", "rows", "rows", "batch", "serve", "pieces", "product",
                        "noalloc"])
        if k == "search":
            c = {"kind": k, "pmin": log(200, 3e9), "width": log(100, 1e6), "fresh": rng.random() < 0.4}
        elif k == "past":
            c = {"kind": "search", "pmin": log(9e9, 4e10), "width": log(200, 1000), "fresh": False}
        elif k == "rows":
            c = {"kind": k, "pmin": log(1e8, TOP - 4e6), "width": log(200, 2e5), "q_cap": log(2 ** 16, 2 ** 29)}
        elif k == "batch":
            c = {"kind": k, "ranges": log(4, 128), "width": log(1000, 30000), "q_cap": log(2 ** 18, 2 ** 26)}
        elif k == "serve":
            c = {"kind": k, "ranges": log(4, 128), "width": log(500, 4000), "q_cap": log(2 ** 18, 2 ** 25)}
        elif k == "pieces":
            c = {"kind": k, "pmin": log(1e5, 1e9), "width": log(1000, 300000), "cut": log(2 ** 8, 2 ** 25)}
        elif k == "product":
            c = {"kind": k, "rows": log(100, 60000), "parts": rng.randrange(2, 9), "bits": rng.randrange(20, 62)}
        else:
            c = {"kind": k, "rows": rng.randrange(1, 4000), "bits": rng.randrange(28, 62),
                 "q_cap": log(2 ** 14, 2 ** 24)}
        if _cost(c) <= 2.5e11:
            return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _sieve(n):
    s = np.ones(n, dtype=bool)
    s[:2] = False
    s[4::2] = False
    for q in range(3, int(n ** 0.5) + 1, 2):
        if s[q]:
            s[q * q::2 * q] = False
    return np.nonzero(s)[0]


def _odd_moduli(n, bits, r):
    """n odd numbers of `bits` bits with no prime factor below 30, which is all that the row arithmetic asks
    of a modulus here."""
    out = r.integers(2 ** (bits - 1), 2 ** bits - 2 ** (bits // 2), 8 * n + 64, dtype=np.int64) | 1
    for q in (3, 5, 7, 11, 13, 17, 19, 23, 29):
        out = out[out % q != 0]
    return np.ascontiguousarray(out[:n].astype(np.uint64))


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "noalloc":
        r = np.random.default_rng(seed)
        p = np.sort(_odd_moduli(case["rows"], case["bits"], r))
        q = _sieve(case["q_cap"])
        s["lib"] = wl.load_library()
        s["bound"] = 2 ** case["bits"]
        s["T"] = (int(p[0]) - 1) // 6
        q = q[q <= s["T"]]
        s["p"] = torch.from_numpy(p.astype(np.int64)).cuda()
        s["q"] = torch.from_numpy(q.astype(np.int32)).cuda()
        s["out"] = torch.empty(2 * len(p), dtype=torch.int64, device="cuda")
        return s
    if kind == "serve":
        s["ranges"] = _ranges(case, seed)
        s["server"] = wl.Server(0)
        return s
    s["engine"] = wl.Engine(0)
    if kind == "batch":
        s["ranges"] = _ranges(case, seed)
    elif kind == "product":
        r = np.random.default_rng(seed)
        s["p"] = _odd_moduli(case["rows"], case["bits"], r)
        s["parts"] = [np.stack([r.integers(0, s["p"], dtype=np.uint64), r.integers(0, s["p"], dtype=np.uint64)], axis=1)
                      for _ in range(case["parts"])]
    else:
        s["range"] = _place(case, seed)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _signed(v):
    return ctypes.c_int64(v).value


def _fields(rows, n, names=("p", "s0", "s1", "rem", "quot")):
    out = {f: np.zeros(n, dtype=np.int64) for f in names}
    for f in names:
        out[f][:len(rows)] = rows[f].view(np.int64)
    return out


def _odd_in(width):
    """As many test primes as a range of this width can hold."""
    return width // 2 + 1


def _lines(results, width):
    out = np.zeros((min(_odd_in(width), 4096), 2), dtype=np.int64)
    if results:
        out[:len(results)] = results
    return out


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "search":
        e = s["engine"]
        if c["fresh"]:
            e.drop_columns()
        r = e.search(*s["range"])
        return {"lines": _lines(r.results, c["width"]), "checksum": _signed(r.checksum), "pi": r.stats.pi_maxtarget}
    if kind == "rows":
        rows, _ = s["engine"].rows(*s["range"], q_cap=c["q_cap"])
        return _fields(rows, _odd_in(c["width"]))
    if kind == "batch":
        per, results, _ = s["engine"].batch(s["ranges"], q_cap=c["q_cap"])
        return {"tested": np.array([x["tested"] for x in per], dtype=np.int64),
                "checksum": np.array([_signed(x["checksum"]) for x in per], dtype=np.int64),
                "targets": np.array([x["targets"] for x in per], dtype=np.int64), "lines": _lines(results, 0)}
    if kind == "serve":
        srv = s["server"]
        ids = [srv.submit(a, b, q_cap=c["q_cap"]) for a, b in s["ranges"]]
        sums, parts = [], []
        for i in ids:
            sums.append(_signed(srv.wait(i).checksum))
            parts.append(srv.rows(i))
            srv.release(i)
        n = sum(_odd_in(b - a) for a, b in s["ranges"])
        return {"checksum": np.array(sums, dtype=np.int64), "rows": _fields(np.concatenate(parts), n)}
    if kind == "pieces":
        e = s["engine"]
        first, _ = e.rows_from(*s["range"], 2, c["cut"])
        r = e.search_from(*s["range"], c["cut"], init=first)
        return {"first": _fields(first, _odd_in(c["width"]), ("p", "s0", "s1")), "lines": _lines(r.results, c["width"]),
                "checksum": _signed(r.checksum)}
    if kind == "product":
        return _fields(s["engine"].rows_product(s["parts"], p=s["p"]), c["rows"], ("p", "s0", "s1"))
    rc = s["lib"].wl_column_product_noalloc(s["p"].data_ptr(), len(s["p"]), s["bound"], s["T"], s["q"].data_ptr(),
                                            len(s["q"]), s["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    if rc:
        raise wl.WilsonError(rc, "wl_column_product_noalloc")
    return s["out"]


def work(case):
    """A multiplication and an addition for each (row, column) pair; the inputs and results once each."""
    k = case["kind"]
    if k in ("search", "pieces"):
        n, cells = _rows(case["pmin"], case["width"]), _cells(case["pmin"], case["width"])
    elif k == "rows":
        n, cells = _rows(case["pmin"], case["width"]), _cells(case["pmin"], case["width"], case["q_cap"])
    elif k in ("batch", "serve"):
        rs = _ranges(case, 0)
        n = sum(_rows(a, b - a) for a, b in rs)
        cells = sum(_cells(a, b - a, case["q_cap"]) for a, b in rs)
    elif k == "product":
        n, cells = case["rows"] * (case["parts"] + 1), case["rows"] * case["parts"]
    else:
        n, cells = case["rows"], case["rows"] * _pi(case["q_cap"])
    return {"bytes": 48.0 * n, "flops": 2.0 * cells}


# ---------------------------------------------------------------------------
# the values, from Python integers
# ---------------------------------------------------------------------------

def _target(p):
    return (p - 1) // 6 if p % 3 == 1 else (p - 1) // 4 if p % 12 == 5 else (p - 1) // 2


def _class(p):
    return 0 if p % 3 == 1 else 1 if p % 12 == 5 else 2


def _exponent(T, q):
    e = 0
    while T:
        T //= q
        e += T
    return e


def _product_mod(qs, T, n):
    x = 1
    for q in qs:
        x = x * pow(q, _exponent(T, q), n) % n
    return x


def _is_prime(n):
    if n < 2:
        return False
    for q in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37):
        if n % q == 0:
            return n == q
    d, s = n - 1, 0
    while d % 2 == 0:
        d, s = d // 2, s + 1
    for a in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37):
        x = pow(a, d, n)
        if x in (1, n - 1):
            continue
        for _ in range(s - 1):
            x = x * x % n
            if x == n - 1:
                break
        else:
            return False
    return True


def _i64(v):
    return np.array(v, dtype=np.uint64).view(np.int64)


def _factorial_mod(p):
    n, x = p * p, 1
    for k in range(2, p):
        x = x * k % n
    return x


def exact(case, seed):
    k = case["kind"]
    if k == "product":
        r = np.random.default_rng(seed)
        p = _odd_moduli(case["rows"], case["bits"], r)
        parts = [(r.integers(0, p, dtype=np.uint64), r.integers(0, p, dtype=np.uint64)) for _ in range(case["parts"])]
        s0, s1 = [], []
        for i, v in enumerate(int(x) for x in p):
            x = 1
            for d0, d1 in parts:
                x = x * (int(d0[i]) + v * int(d1[i])) % (v * v)
            s0.append(x % v)
            s1.append(x // v)
        return {"p": p.view(np.int64), "s0": _i64(s0), "s1": _i64(s1)}
    if k == "noalloc" and case["rows"] * _pi(case["q_cap"]) <= 2e6:
        r = np.random.default_rng(seed)
        p = np.sort(_odd_moduli(case["rows"], case["bits"], r))
        T = (int(p[0]) - 1) // 6
        qs = [int(q) for q in _sieve(case["q_cap"]) if q <= T]
        out = []
        for v in (int(x) for x in p):
            x = _product_mod(qs, T, v * v)
            out += [x % v, x // v]
        return torch.from_numpy(_i64(out))
    if k == "rows" and case["q_cap"] and _cells(case["pmin"], case["width"], case["q_cap"]) <= 1e6:
        a, b = _place(case, seed)
        ps = [p for p in range(a, b) if _is_prime(p)]
        T = {}
        for p in ps:
            T.setdefault(_class(p), _target(p))
        qs = [int(q) for q in _sieve(case["q_cap"])]
        s0, s1 = [], []
        for p in ps:
            t = T[_class(p)]
            x = _product_mod([q for q in qs if q <= t], t, p * p)
            s0.append(x % p)
            s1.append(x // p)
        n = _odd_in(case["width"])
        pad = lambda v: np.concatenate([_i64(v), np.zeros(n - len(v), dtype=np.int64)])
        return {"p": pad(ps), "s0": pad(s0), "s1": pad(s1), "rem": pad([]), "quot": pad([])}
    if k == "search" and case["pmin"] * _rows(case["pmin"], case["width"]) <= 1e7:
        a, b = _place(case, seed)
        ps = [p for p in range(a, b) if _is_prime(p)]
        lines, check, top = [], 0, 0
        for p in ps:
            x = (_factorial_mod(p) + 1) % (p * p)
            rem, quot = x % p, x // p
            check += p + rem + quot
            if min(quot, p - quot) < 1000:
                lines.append((p, quot if quot <= p - quot else quot - p))
        for c in range(3):
            first = [p for p in ps if _class(p) == c][:1]
            top = max([top] + [_target(p) for p in first])
        return {"lines": _lines(lines, b - a), "checksum": _signed(check & (2 ** 64 - 1)), "pi": len(_sieve(top + 1))}
    return None
