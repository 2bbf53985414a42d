"""CPU model of the integer bookkeeping of a divide-and-conquer level (csrc/tridiag_quadrature.cu:
dc_sorted_merge, dc_next, dc_drop_rank, dc_merged_place), element by element as its threads do it:
the sorted positions of the two halves, negligible and close poles moved behind the kept ones, and
the places of roots and dropped poles in the merged order.

Every position is written once, kept and dropped poles are those of a sequential deflation, and a
column index that is followed names a column, whatever the values: NaN leaves the poles of a half
unordered, two elements then take one position, and the position left over keeps what it had."""

import math
import random
import struct

import pytest

EPS = 2.0 ** -52
LIVE, CLOSE, GONE = 1, 2, 4


def key(x):
    v = struct.unpack("<q", struct.pack("<d", x))[0]
    return v ^ ((v >> 63) & 0x7FFFFFFFFFFFFFFF)


def nxt(O, r, hi):
    r += 1
    while r < hi and O[r] == 0:
        r += 1
    return r


def merge(LAM, Z0, EO, k, s, D, Z, CI):
    """One level; Z0[r]: weight of element r.  Returns (kept counts, flips) per merge."""
    w = 1 << s
    nm = (k - w - 1) // (2 * w) + 1
    written = set()
    for r in range(k):
        q = r >> (s + 1)
        if q >= nm:
            continue
        a = q * 2 * w
        mid, hi = a + w, min(a + 2 * w, k)
        flip, first = EO[mid - 1] < 0.0, r < mid
        own = ((mid - 1 - r if first else hi - 1 - r) if flip else (r - a if first else r - mid))
        v = -LAM[r] if flip else LAM[r]
        lo, up = 0, (hi - mid if first else w)
        while lo < up:
            c = (lo + up) >> 1
            i = (hi - 1 - c if flip else mid + c) if first else (mid - 1 - c if flip else a + c)
            other = key(-LAM[i] if flip else LAM[i])
            if other < key(v) if first else other <= key(v):
                lo = c + 1
            else:
                up = c
        pos = a + own + lo
        assert a <= pos < hi
        written.add(pos)
        D[pos], Z[pos], CI[pos] = v, Z0[r], r
    rho = [abs(EO[q * 2 * w + w - 1]) for q in range(nm)]
    span = [(q * 2 * w, min(q * 2 * w + 2 * w, k)) for q in range(nm)]
    tol = [8.0 * EPS * max(abs(D[a]), abs(D[hi - 1]), 2.0 * rho[q]) for q, (a, hi) in enumerate(span)]
    O = [0] * k
    for q, (a, hi) in enumerate(span):
        for r in range(a, hi):
            O[r] = 0 if rho[q] * abs(Z[r]) <= tol[q] else LIVE
    for q, (a, hi) in enumerate(span):
        for r in range(a, hi):
            if O[r] == 0:
                continue
            prev = r - 1
            while prev >= a and O[prev] == 0:
                prev -= 1
            if prev >= a and D[r] - D[prev] <= tol[q]:
                O[r] = LIVE | CLOSE
    for q, (a, hi) in enumerate(span):
        for r in range(a, hi):
            if O[r] & (LIVE | CLOSE) != LIVE:
                continue
            p, n = r, nxt(O, r, hi)
            while n < hi and O[n] & CLOSE:
                Z[n] = math.hypot(Z[p], Z[n])
                O[p] |= GONE
                p, n = n, nxt(O, n, hi)
    counts = []
    for q, (a, hi) in enumerate(span):
        kept = [r for r in range(a, hi) if O[r] and not O[r] & GONE]
        order = [0] * (hi - a)
        for r in range(a, hi):
            before = sum(1 for i in kept if i < r)
            at = before if r in kept else len(kept) + (r - a - before)
            order[at] = r
        D[a:hi], Z[a:hi], CI[a:hi] = [D[r] for r in order], [Z[r] for r in order], [CI[r] for r in order]
        counts.append(len(kept))
    return counts, [EO[a + w - 1] < 0.0 for a, _ in span], span, written


def places(X, D, a, mk, hi, flip):
    """Position of element r of a merge among the roots X[a : a + mk] and dropped poles D[a + mk : hi]."""
    C = {r: sum(1 for i in range(a, a + mk) if key(X[i]) <= key(D[r])) for r in range(a + mk, hi)}
    out = {}
    for r in range(a, hi):
        j = r - a
        at = j - mk + C[r] if j >= mk else j + sum(1 for c in C.values() if c <= j)
        out[r] = hi - 1 - at if flip else a + at
    return out


def roots(D, Z, a, mk, rho):
    """Stand-ins that interlace as the secular roots do."""
    out = []
    for j in range(mk):
        up = D[a + j + 1] if j + 1 < mk else D[a + j] + 2.0 * rho + 1.0
        out.append(fp(0.5 * (D[a + j] + up)))
    return out


def fp(x):
    """The device's arithmetic gives one NaN, of positive sign; a negation turns its sign."""
    return math.nan if math.isnan(x) else x


def run(k, rng, special=None, columns=None, one_zero=True):
    scale = 10.0 ** rng.randint(-3, 3)
    LAM = [scale * rng.choice([0.0, 1.0, rng.random(), 1.0 + EPS * rng.randint(0, 9)]) for _ in range(k)]
    EO = [scale * rng.choice([0.0, 1e-18, 0.3, -0.3, rng.random() - 0.5]) for _ in range(k)]
    if special is not None:
        for _ in range(2):
            LAM[rng.randrange(k)] = special * rng.choice([1.0, -1.0])
    D, Z = [0.0] * k, [0.0] * k
    CI = list(range(k)) if columns is None else columns
    for s in range(20):
        if 1 << s >= k:
            break
        Z0 = [rng.choice([1e-20, 1.0, 0.1, rng.random()]) for _ in range(k)]
        before = list(LAM)
        counts, flips, span, written = merge(LAM, Z0, EO, k, s, D, Z, CI)
        for q, (a, hi) in enumerate(span):
            assert all(0 <= c < k for c in CI[a:hi])  # a column is a column
            if special is None:
                assert all(p in written for p in range(a, hi))
                assert sorted(CI[a:hi]) == list(range(a, hi))
                sg = -1.0 if flips[q] else 1.0
                assert sorted(D[a:hi]) == sorted(sg * x for x in before[a:hi])
                mk = counts[q]
                assert D[a:a + mk] == sorted(D[a:a + mk]) and D[a + mk:hi] == sorted(D[a + mk:hi])
                assert all(y > x for x, y in zip(D[a:a + mk], D[a + 1:a + mk]))
            X = {a + j: x for j, x in enumerate(roots(D, Z, a, counts[q], abs(EO[a + (1 << s) - 1])))}
            at = places(X, D, a, counts[q], hi, flips[q])
            assert all(a <= p < hi for p in at.values())
            new = list(LAM)
            for r, p in at.items():
                v = X[r] if r in X else D[r]
                new[p] = -v if flips[q] else v
                if one_zero:
                    new[p] = fp(new[p] + 0.0)
            LAM[a:hi] = new[a:hi]
            if special is None:
                assert sorted(at.values()) == list(range(a, hi))
                assert [key(x) for x in LAM[a:hi]] == sorted(key(x) for x in LAM[a:hi])


@pytest.mark.parametrize("k", [2, 3, 16, 17, 31, 33, 48, 64])
def test_level_bookkeeping(k):
    rng = random.Random(k)
    for _ in range(40):
        run(k, rng)


@pytest.mark.parametrize("special", [math.nan, math.inf])
@pytest.mark.parametrize("k", [16, 17, 33, 48])
def test_columns_stay_columns_with_special_values(k, special):
    rng = random.Random(k)
    for _ in range(60):
        run(k, rng, special)


def test_what_happens_without_the_start_value_and_the_sum():
    """The index array as shared memory holds it at first, and negated values as they are: some NaN
    has a word followed that no element wrote."""
    rng, seen = random.Random(5), 0
    for _ in range(200):
        try:
            run(17, rng, math.nan, columns=[1 << 30] * 17, one_zero=False)
        except AssertionError:
            seen += 1
    assert seen > 0


def _sequential(items, rho, tol):
    """The deflation one pole after the other: kept (value, weight) and dropped values."""
    kept, dropped = [], []
    for d, z in items:
        if rho * abs(z) <= tol:
            dropped.append(d)
        elif kept and d - kept[-1][0] <= tol:
            dropped.append(kept[-1][0])
            kept[-1] = (d, math.hypot(kept[-1][1], z))
        else:
            kept.append((d, z))
    return kept, sorted(dropped)


@pytest.mark.parametrize("seed", range(30))
def test_deflation_is_the_sequential_one(seed):
    rng = random.Random(seed)
    k = 32
    base = sorted(rng.choice([0.0, 1.0, 2.0]) + 4.0 * EPS * rng.randint(0, 12) for _ in range(16))
    other = sorted(rng.choice([0.0, 1.0, 2.0]) + 4.0 * EPS * rng.randint(0, 12) for _ in range(16))
    LAM, EO = base + other, [0.0] * k
    EO[15] = rng.choice([0.4, 1e-3])
    Z0 = [rng.choice([1e-20, 0.2, rng.random()]) for _ in range(k)]
    D, Z, CI = [0.0] * k, [0.0] * k, list(range(k))
    counts, _, _, _ = merge(LAM, Z0, EO, k, 4, D, Z, CI)
    order = sorted(range(k), key=lambda r: (LAM[r], r))
    tol = 8.0 * EPS * max(abs(min(LAM)), abs(max(LAM)), 2.0 * EO[15])
    kept, dropped = _sequential([(LAM[r], Z0[r]) for r in order], EO[15], tol)
    mk = counts[0]
    assert [(D[i], Z[i]) for i in range(mk)] == kept
    assert D[mk:] == dropped
