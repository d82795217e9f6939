"""The complex modular products in rings where -1 is a square (csrc/oz_ring.cu), restated on the CPU.

* the moduli: pairwise coprime, i_m with i_m^2 = -1 exists, enough of them for every plan;
* the split: residues of x +- i_m y by byte dot products started at FP32 bits, at the extremes of x, y;
* the products and their recombination, two moduli at a time, against exact integers (the error bound is
  the rounding of the pair constants plus one unit of the 64-bit window);
* the flat (tile, plane) work list: every product exactly once, for few and many tiles per cluster.
"""
import ctypes
import math

import numpy as np
import pytest

from exciting_b200 import abi

RINGS = [241, 233, 229, 221, 205, 197, 193, 181, 173, 157, 149, 137, 113, 109, 101, 97]


def bits_of_plan(n):
    lib = abi.load()
    b, bx = ctypes.c_int(), ctypes.c_int()
    assert lib.exs_ozaki_moduli(n, 1936, 242, None, None, None, ctypes.byref(b), ctypes.byref(bx), None) == 0
    return b.value, bx.value


def rings(b, bx):
    want, lm, out = max(2 * b, b + bx) + 2, 0.0, []
    for p in RINGS:
        if lm - 1e-9 >= want:
            break
        out.append(p)
        lm += math.log2(p)
    assert lm - 1e-9 >= want
    return out, lm


def root(p):
    return next(i for i in range(p) if (i * i + 1) % p == 0)


def sym(v, p):
    v %= p
    return v - p if v > p // 2 else v


@pytest.mark.parametrize("n", range(6, 17))
def test_rings_hold_every_plan(n):
    b, bx = bits_of_plan(n)
    ps, _ = rings(b, bx)
    M = math.prod(ps)
    assert M >= 2 ** (2 * b + 2) and M >= 2 ** (b + bx + 2)
    for i, p in enumerate(ps):
        assert (root(p) ** 2 + 1) % p == 0 and p <= 254
        assert all(math.gcd(p, q) == 1 for q in ps[:i])
    if n == 13:
        assert len(ps) == 14


def split(x, y, p):
    """int64 arrays x, y (|.| <= 2^52) -> residue bytes of x + i y and x - i y, in the kernel's arithmetic."""
    im, f32 = root(p), np.float32
    dig = lambda v: [((v + (1 << 55)) >> (8 * k)) & 255 for k in range(7)]  # noqa: E731
    off = -((1 << 55) % p)
    start = 12582912 // p * p
    vr = start + sym(off, p) + sum(d * sym(1 << (8 * k), p) for k, d in enumerate(dig(x)))
    vi = sym(off * im, p) + sum(d * sym((1 << (8 * k)) * im, p) for k, d in enumerate(dig(y)))
    out = []
    for v in (vr + vi, vr - vi):
        assert v.min() >= 2 ** 23 and v.max() < 2 ** 24                 # an FP32 integer with unit ulp
        inv = np.float64(f32(1.0) / f32(p))
        q = (v * inv + 12582912.0).astype(f32).astype(np.int64) - 12582912      # exact product, one rounding
        r = v - q * p
        assert np.abs(r).max() <= 127
        out.append(((v - q * p) & 255).astype(np.uint8).view(np.int8).astype(np.int64))
        assert np.array_equal(out[-1], r)
    return out


@pytest.mark.parametrize("p", RINGS)
def test_split_residues(p):
    rng = np.random.default_rng(p)
    ends = np.array([0, 1, -1, 2 ** 52, -2 ** 52, 2 ** 51, -2 ** 49 - 1], dtype=np.int64)
    x = np.concatenate([rng.integers(-2 ** 52, 2 ** 52, 5000), np.repeat(ends, ends.size)])
    y = np.concatenate([rng.integers(-2 ** 52, 2 ** 52, 5000), np.tile(ends, ends.size)])
    s, d = split(x, y, p)
    im = root(p)
    assert all((int(a) + im * int(c) - int(r)) % p == 0 for a, c, r in zip(x, y, s))
    assert all((int(a) - im * int(c) - int(r)) % p == 0 for a, c, r in zip(x, y, d))


def reduce(v, p):
    """The byte the short product kernel stores for the int32 sums v, |v| < 2^27."""
    x = v + ((1 << 27) // p + 1) * p
    r = x - ((x * ((1 << 32) // p)) >> 32) * p
    assert r.min() >= 0 and r.max() <= 246
    return r


@pytest.mark.parametrize("p", RINGS)
def test_short_reduction(p):
    """Bytes congruent to the sums over the whole range of the short kernel."""
    v = np.concatenate([np.random.default_rng(p).integers(-2 ** 27 + 1, 2 ** 27, 20000),
                        np.array([0, -1, 1, p, -p, p - 1, -p - 1, 2 ** 27 - 1, -2 ** 27 + 1])])
    assert np.array_equal(reduce(v, p) % p, v % p)
    assert 8192 * 123 ** 2 < 2 ** 27


@pytest.mark.parametrize("n", [6, 13, 14, 16])
def test_products_recombine(n):
    """conj(A)^T B of integer columns of norm 2^b, through the rings."""
    b, bx = bits_of_plan(n)
    ps, lm = rings(b, bx)
    M = math.prod(ps)
    rng = np.random.default_rng(n)
    K = 90
    Z = rng.standard_normal((2, K, 4)) + 1j * rng.standard_normal((2, K, 4))
    Z *= 2.0 ** b * (1 - 1e-9) / np.linalg.norm(Z, axis=1, keepdims=True)
    Z[1, :, 0] = -Z[0, :, 0]                                            # the bound's extreme
    ar, ai = np.trunc(Z[0].real).astype(np.int64), np.trunc(Z[0].imag).astype(np.int64)
    br, bi = np.trunc(Z[1].real).astype(np.int64), np.trunc(Z[1].imag).astype(np.int64)
    sh = max(0, min(20, math.floor(lm - 1e-9 - 2 * b - 3)))
    t = np.zeros((2, 4, 4), dtype=object)
    bound = 0
    for q in range(0, len(ps), 2):
        pair = ps[q:q + 2]
        pq = math.prod(pair)
        w = np.full((2, 4, 4), -(-(1 << 26) // pq) * pq, dtype=object)
        for j, p in enumerate(pair):
            (ap, am), (bp, bm) = split(ar, ai, p), split(br, bi, p)
            zp, zm = reduce(am.T @ bp, p), reduce(ap.T @ bm, p)         # exact: K 127^2 < 2^27
            y, half, other = pow(M // p, -1, p), pow(2, -1, p), pq // p
            for c, f in ((0, y * half % p * other), (1, y * half % p * pow(root(p), -1, p) % p * other)):
                f -= pq if f > pq // 2 else 0
                for sgn in (1, -1):                                     # two signed bytes hold +-f
                    lo = sym(sgn * f, 256) if sym(sgn * f, 256) < 128 else -128
                    assert -128 <= (sgn * f - lo) // 256 <= 127
                w[c] += f * (zp + (-1) ** c * zm).astype(object)
        assert w.min() >= 0 and w.max() < 2 ** 27
        t += w * ((((1 << (96 + sh)) + pq // 2) // pq) % 2 ** 96)
        bound += 2 ** 27 / 2
    for part, exact in ((0, lambda i, j: ar[:, i].astype(object) @ br[:, j] + ai[:, i].astype(object) @ bi[:, j]),
                        (1, lambda i, j: ar[:, i].astype(object) @ bi[:, j] - ai[:, i].astype(object) @ br[:, j])):
        for i in range(4):
            for j in range(4):
                top = (int(t[part, i, j]) >> 32) % 2 ** 64
                top -= 2 ** 64 if top >= 2 ** 63 else 0
                err = abs(top * M - int(exact(i, j)) * 2 ** (64 + sh))
                assert err <= (bound / 2 ** 32 + 1) * M


@pytest.mark.parametrize("runs", [False, True])
@pytest.mark.parametrize("ntiles,ncl,planes", [(1, 28, 28), (2, 56, 28), (3, 74, 28), (74, 74, 28), (75, 74, 28),
                                               (147, 74, 30), (540, 74, 28)])
def test_work_list_covers_every_product_once(ntiles, ncl, planes, runs):
    full = ntiles // ncl
    full_end = full * ncl
    rest = ntiles - full_end
    pairs = rest * planes
    seen, most, least = set(), 0, 1 << 30
    for c in range(ncl):
        first = pairs * c // ncl if runs else c
        mine = pairs * (c + 1) // ncl - first if runs else (pairs - c + ncl - 1) // ncl
        count = full * planes + mine
        most, least = max(most, count), min(least, count)
        start = (full_end + first // planes, first % planes) if runs else (full_end + first % max(rest, 1),
                                                                           first // max(rest, 1))
        tile, P = (c, 0) if full else start
        for _ in range(count):
            assert (tile, P) not in seen and tile < ntiles and P < planes
            seen.add((tile, P))
            if tile >= full_end:
                if runs:
                    tile, P = (tile, P + 1) if P + 1 < planes else (tile + 1, 0)
                else:
                    v = tile - full_end + ncl
                    tile, P = full_end + v % rest, P + v // rest
            else:
                tile, P = (tile, P + 1) if P + 1 < planes else (tile + ncl, 0)
                if tile >= full_end:
                    tile, P = start
    assert len(seen) == ntiles * planes and most - least <= 1
