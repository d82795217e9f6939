"""The constants and the work list that the modular products run with, as the library's own code forms them.

csrc/oz_ring.cu is compiled into a host program that prints oz_ring_plan's constants (packed weights,
offsets, reciprocals, windows) and walks RingUnits.  The device arithmetic is then carried out on the CPU
with those values: the split of b-bit integers into residues, the products, both reductions of the int32
sums and the recombination, for the H/O products and for the per-atom products of every plan, against exact
integers.
"""
import ctypes
import math
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from exciting_b200 import abi, build
from exciting_b200.fvsystem import ozaki_moduli, ozaki_rings

K, KX = 1936, 242
LISTS = [(1, 28, 28), (2, 56, 28), (3, 74, 28), (74, 74, 28), (75, 74, 28), (147, 74, 30), (540, 74, 26)]

SOURCE = r"""
#include <cstdio>
#include "oz_ring.cu"
using namespace exs;

static void crt(const OzCrt &c)
{
    std::printf("%d %d %a", c.n, c.sh, c.fin);
    for (int q = 0; q < OZ_RING_MAX / 2; q++) {
        std::printf(" %d", c.woff[q]);
        for (int k = 0; k < 2; k++) std::printf(" %d %d", c.wlo[k][q], c.whi[k][q]);
        for (int w = 0; w < 3; w++) std::printf(" %u", c.d96[w][q]);
    }
    std::printf("\n");
}

template <bool RUNS>
static void walk(int ntiles, int ncl, int np)
{
    std::printf("%d %d %d %d", (int)RUNS, ntiles, ncl, np);
    for (int c = 0; c < ncl; c++) {
        RingUnits<RUNS> u(ntiles, ncl, np, c);
        std::printf(" %d", -u.count);
        for (int i = 0; i < u.count; i++, u.next()) std::printf(" %d %d", u.tile, u.P);
    }
    std::printf("\n");
}

int main()
{
    for (int n = 6; n <= 16; n++) {
        OzScheme s{};
        OzRing r{};
        if (oz_mod_plan(n, K_, KX_, &s) || oz_ring_plan(s.b, s.bx, &r)) return 1;
        std::printf("%d %d %d\n", r.n, r.b, r.bx);
        for (int m = 0; m < r.n; m++)
            std::printf("%d %d %u %d %a %d %d %d %d %d %d\n", r.p[m], r.mg[m], r.mf[m], r.up[m], (double)r.inv[m],
                        r.clo[m], r.chi[m], r.ilo[m], r.ihi[m], r.base[m], r.icorr[m]);
        crt(r.ho);
        crt(r.at);
    }
    const int lists[][3] = {LISTS_};
    for (auto &l : lists) {
        walk<false>(l[0], l[1], l[2]);
        walk<true>(l[0], l[1], l[2]);
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def dump(tmp_path_factory):
    d = tmp_path_factory.mktemp("rings")
    src = SOURCE.replace("KX_", str(KX)).replace("K_", str(K))
    src = src.replace("LISTS_", ", ".join("{%d, %d, %d}" % l for l in LISTS))
    (d / "rings.cu").write_text(src)
    flags = [f for f in build.FLAGS if f not in ("-shared", "-lineinfo", "-O3")]
    subprocess.run([build.nvcc(), *build.ARCH, *flags, "-O1", "-I", build.CSRC, "-o", str(d / "rings"),
                    str(d / "rings.cu")], check=True)
    lines = subprocess.run([str(d / "rings")], check=True, capture_output=True, text=True).stdout.splitlines()
    it, plans = iter(lines), {}
    num = lambda t: float.fromhex(t) if "0x" in t else int(t)  # noqa: E731
    for n in range(6, 17):
        cnt, b, bx = (int(x) for x in next(it).split())
        keys = ("p", "mg", "mf", "up", "inv", "clo", "chi", "ilo", "ihi", "base", "icorr")
        rows = [dict(zip(keys, (num(t) for t in next(it).split()))) for _ in range(cnt)]
        crts = []
        for _ in range(2):
            v = [num(t) for t in next(it).split()]
            pairs = [v[3 + 8 * q: 11 + 8 * q] for q in range(8)]
            crts.append(dict(n=v[0], sh=v[1], fin=v[2], pairs=pairs))
        plans[n] = dict(b=b, bx=bx, rings=rows, ho=crts[0], at=crts[1])
    return plans, [[int(x) for x in line.split()] for line in it]


def signed_bytes(w):
    return [int(np.int8(np.uint8((w >> (8 * k)) & 255))) for k in range(4)]


def dp4a(bytes_u, w, c):
    """Unsigned bytes (four arrays) times the signed bytes of the word w."""
    return sum(x * y for x, y in zip(bytes_u, signed_bytes(w))) + c


def split(x, y, r):
    """Residue bytes of x + i y and x - i y, |x|, |y| <= 2^52 (int64 arrays), by ring_pair's steps."""
    dig = lambda v: [((v + (1 << 55)) >> (8 * k)) & 255 for k in range(8)]  # noqa: E731
    dx, dy = dig(x), dig(y)
    vr = dp4a(dx[:4], r["clo"], dp4a(dx[4:], r["chi"], r["base"]))
    vi = dp4a(dy[:4], r["ilo"], dp4a(dy[4:], r["ihi"], r["icorr"]))
    out = []
    for v in (vr + vi, vr - vi):
        f = v.astype(np.int32).view(np.float32)
        assert f.min() >= 2.0 ** 23 and f.max() < 2.0 ** 24
        q = (f.astype(np.longdouble) * np.longdouble(r["inv"]) + np.longdouble(12582912.0)).astype(np.float32)
        byte = (v - q.view(np.int32).astype(np.int64) * r["p"]) & 255
        out.append(byte.astype(np.uint8).view(np.int8).astype(np.int64))
    return out


def reduce_short(v, r):
    x = v + r["up"]
    assert x.min() >= 0 and x.max() < 2 ** 32
    z = x - ((x * r["mf"]) >> 32) * r["p"]
    assert z.min() >= 0 and z.max() <= 255
    return z


def reduce_long(v, r):
    assert np.abs(v).max() < 2 ** 30
    x = (v - ((v * r["mg"]) >> 32) * r["p"]) % 2 ** 32
    x = np.minimum(x, (x + r["p"]) % 2 ** 32)
    return np.minimum(x, (x - r["p"]) % 2 ** 32)


def recombine(c, zp, zm):
    """ring_crt4: real and imaginary values (objects: exact fractions of the double) from the residues."""
    acc = [[0, 0, 0], [0, 0, 0]]
    zero = np.zeros_like(zp[0])
    for q in range((c["n"] + 1) // 2):
        woff, lo0, hi0, lo1, hi1, d0, d1, d2 = c["pairs"][q]
        second = 2 * q + 1 < len(zp)
        z = [zp[2 * q], zm[2 * q], zp[2 * q + 1] if second else zero, zm[2 * q + 1] if second else zero]
        for part, (lo, hi) in enumerate(((lo0, hi0), (lo1, hi1))):
            w = dp4a(z, lo, woff) + 256 * dp4a(z, hi, 0)
            assert w.min() >= 0 and w.max() < 2 ** 27
            w = w.astype(object)
            for k, d in enumerate((d0, d1, d2)):
                acc[part][k] = acc[part][k] + w * d
    out = []
    for a0, a1, a2 in acc:
        assert max(a0.max(), a1.max()) < 2 ** 64
        c1 = a1 + (a0 // 2 ** 32)
        assert c1.max() < 2 ** 64
        top = ((a2 + c1 // 2 ** 32) % 2 ** 32) * 2 ** 32 + c1 % 2 ** 32
        top = np.vectorize(lambda t: t - 2 ** 64 if t >= 2 ** 63 else t, otypes=[object])(top)
        out.append(np.vectorize(lambda t: float(t) * c["fin"], otypes=[object])(top))
    return out


def integers(rng, bits, rows):
    """Integer columns of 2-norm up to 2^bits, one of them with all of it in a single entry."""
    z = rng.standard_normal((rows, 4)) + 1j * rng.standard_normal((rows, 4))
    z *= 2.0 ** bits * (1 - 1e-9) / np.linalg.norm(z, axis=0)
    z[:, 3] = 0.0
    z[rows // 2, 3] = 2.0 ** bits * (1 - 1e-9)
    return np.trunc(z.real).astype(np.int64), np.trunc(z.imag).astype(np.int64)


@pytest.mark.parametrize("n", range(6, 17))
def test_plan_matches_the_query(dump, n):
    d = dump[0][n]
    ps, n_atom = ozaki_rings(n, K, KX)
    _, _, b, bx, _ = ozaki_moduli(n, K, KX)
    assert (d["b"], d["bx"]) == (b, bx) and [r["p"] for r in d["rings"]] == ps
    assert d["ho"]["n"] == len(ps) and d["at"]["n"] == n_atom <= len(ps)
    assert math.prod(ps) >= 2 ** (2 * b + 2) and math.prod(ps[:n_atom]) >= 2 ** (b + bx + 2)
    for i, p in enumerate(ps):
        assert any((x * x + 1) % p == 0 for x in range(p)) and all(math.gcd(p, q) == 1 for q in ps[:i])


def test_query_rejects_what_the_plan_rejects():
    lib = abi.load()
    out = ctypes.c_int()
    for args in ((5, K, KX), (17, K, KX), (14, 70000, KX), (14, 0, KX), (14, K, 0)):
        assert lib.exs_ozaki_rings(*args, ctypes.byref(out), None, None) < 0
    assert lib.exs_ozaki_rings(13, K, KX, ctypes.byref(out), None, None) == 0 and out.value == 14


@pytest.mark.parametrize("short", [True, False])
@pytest.mark.parametrize("kind", ["ho", "at"])
@pytest.mark.parametrize("n", range(6, 17))
def test_library_constants_reproduce_exact_products(dump, n, kind, short):
    """conj(A)^T B with b-bit columns (H, O), h A with bx-bit rows of h (per-atom products)."""
    d = dump[0][n]
    rng = np.random.default_rng(100 * n + (kind == "at"))
    ar, ai = integers(rng, d["b"], 90)
    br, bi = integers(rng, d["b"] if kind == "ho" else d["bx"], 90)
    c = d[kind]
    reduce = reduce_short if short else reduce_long
    zp, zm = [], []
    for r in d["rings"][: c["n"]]:
        ap, am = split(ar, ai, r)
        bp, bm = split(br, bi, r)
        assert all(np.abs(v).max() <= 123 for v in (ap, am, bp, bm))
        if kind == "ho":                                    # plane 2m: A-, B+; plane 2m + 1: A+, B-
            zp.append(reduce(am.T @ bp, r))
            zm.append(reduce(ap.T @ bm, r))
        else:
            zp.append(reduce(ap.T @ bp, r))
            zm.append(reduce(am.T @ bm, r))
    s = 1 if kind == "ho" else -1                           # conj(A) or A
    A, B = [x.astype(object) for x in (ar, ai)], [x.astype(object) for x in (br, bi)]
    exact = (A[0].T @ B[0] + s * (A[1].T @ B[1]), A[0].T @ B[1] - s * (A[1].T @ B[0]))
    bits = 2 * d["b"] if kind == "ho" else d["b"] + d["bx"]
    M = math.prod(r["p"] for r in d["rings"][: c["n"]])
    pairs = (c["n"] + 1) // 2
    # pair constants round to half a unit of 2^-96 with weights below 2^27, the window drops below one unit of
    # 2^-64; the conversion, M in FP64 and the product with it round by 2^-53 each
    unit = Fraction(M, 2 ** (64 + c["sh"])) * (1 + Fraction(pairs * 2 ** 26, 2 ** 32))
    for got, want in zip(recombine(c, zp, zm), exact):
        for g, w in zip(got.ravel(), want.ravel()):
            assert abs(Fraction(g) * 2 ** bits - int(w)) <= unit + abs(int(w)) * Fraction(4, 2 ** 53)


@pytest.mark.parametrize("i", range(2 * len(LISTS)))
def test_work_list_covers_every_product_once(dump, i):
    v = dump[1][i]
    runs, ntiles, ncl, planes = v[:4]
    assert runs == i % 2 and (ntiles, ncl, planes) == LISTS[i // 2]
    pos, seen, counts = 4, set(), []
    for _ in range(ncl):
        counts.append(-v[pos])
        pos += 1
        for _ in range(counts[-1]):
            unit = (v[pos], v[pos + 1])
            pos += 2
            assert unit not in seen and 0 <= unit[0] < ntiles and 0 <= unit[1] < planes
            seen.add(unit)
    assert pos == len(v) and len(seen) == ntiles * planes and max(counts) - min(counts) <= 1
