"""The work that programs have this library do, for timing it and for checking its outputs.

A case is a plain dict.  ``kind`` says which public calls a pass makes:

* ``setup``   -- Setup.setup_batched_device: the k-loop of one SCF iteration, all arrays on the GPU
* ``graph``   -- the same batch as a captured graph, replayed (fixed k-set, inputs rewritten in place)
* ``host``    -- Setup.setup_batched on host arrays: the drop-in form of a host program's k-loop
* ``scf``     -- a whole SCF iteration: hmlint, olprad, set_scf_inputs, then the batch
* ``rt``      -- rttddft_updateham_device: one time step of RT-TDDFT, momentum matrices resident
* ``adjoint`` -- Setup.adjoint: the backward direction, gradients to positions, V(G) and h_a

Cells: ``fcc`` (two-atom diamond) or ``cube`` (n1 x n2 x n3 supercells of the eight-atom diamond
cube, sites displaced at random).  Atom positions, radial functions, integrals, potentials and
vectors come from the seed; the lattice and the k-points, and with them every size, from the case.
"""
import functools
import math

import numpy as np
import torch

from exciting_b200 import workloads as W
from exciting_b200.basis import Basis
from exciting_b200.crystal import Crystal
from exciting_b200.fvsystem import Setup

NSTATES = 40                      # occupied states of the adjoint cases (the force-check recipe)
DEFAULTS = dict(kind="setup", cell="cube", n1=1, n2=1, n3=1, a=10.26, rgkmax=8.0, lmax=8, basis="text",
                rel="none", nk=1, prec="ozaki_mod")


def _case(name=None, **kw):
    c = dict(DEFAULTS, **kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one k-point of the smallest cell in the default precision: latency
        _case("fcc_k1_fp64", cell="fcc", basis="shipped", rgkmax=7.0, prec="fp64"),
        # the irreducible mesh of the two-atom cell, as a graph that an SCF loop replays
        _case("fcc_k8_mod_graph", kind="graph", cell="fcc", rgkmax=7.0, nk=8),
        # the 27-k batch of the eight-atom cell (rich basis), split precision and native FP64
        _case("cube8_k27_mod", lmax=10, basis="lo3", nk=27),
        _case("cube8_k27_fp64", lmax=10, basis="lo3", nk=27, prec="fp64"),
        # scalar-relativistic overlap terms, smaller cutoff
        _case("cube8_k9_iora_mod", rgkmax=7.0, nk=9, rel="iora*"),
        # mid-size supercell, odd number of k-points
        _case("cube16_k3_zora_mod", n1=2, nk=3, rel="zora"),
        # the largest: one k-point of a 64-atom supercell, and a 32-atom one in native FP64
        _case("cube64_k1_mod", n1=2, n2=2, n3=2),
        _case("cube32_k1_fp64", n1=2, n2=2, prec="fp64"),
        # a host program's call: H and O come back to its own (pageable) arrays
        _case("cube8_k4_mod_host", kind="host", lmax=10, basis="lo3", nk=4),
        # gradients of the setup for 40 states
        _case("cube8_adjoint", kind="adjoint", lmax=10, basis="lo3"),
        # RT-TDDFT time step over the 27-k batch
        _case("cube8_k27_rt_mod", kind="rt", lmax=10, basis="lo3", nk=27),
        # a whole SCF iteration of the eight-atom cell
        _case("cube8_k8_scf_mod", kind="scf", lmax=10, basis="lo3", nk=8),
    ]


def draw(rng):
    kind = rng.choice(["setup"] * 5 + ["graph", "host", "adjoint", "rt", "scf"])
    prec = rng.choice(["ozaki_mod", "ozaki_mod", "ozaki_mod", "fp64"])
    rel = rng.choice(["none", "none", "zora", "iora*"])
    if rng.random() < 0.3:        # two-atom cells of the uneven batch: a and the cutoff vary
        c = _case(kind=kind, cell="fcc", a=round(rng.uniform(9.8, 10.8), 3), rgkmax=round(rng.uniform(6.0, 9.0), 2),
                  basis=rng.choice(["shipped", "text"]), nk=rng.randint(1, 16), prec=prec, rel=rel)
    else:
        n1, n2, n3 = rng.choice([(1, 1, 1), (1, 1, 1), (2, 1, 1), (2, 2, 1), (3, 1, 1), (2, 2, 2)])
        n = n1 * n2 * n3
        nk = {1: rng.randint(1, 27), 2: rng.randint(1, 5), 3: rng.randint(1, 3), 4: 1, 8: 1}[n]
        top = 8.0 if n < 8 else 7.5
        c = _case(kind=kind, n1=n1, n2=n2, n3=n3, a=round(rng.uniform(10.0, 10.4), 3),
                  rgkmax=round(rng.uniform(5.5, top), 2), lmax=rng.choice([8, 8, 9, 10]) if n < 4 else 8,
                  basis=rng.choice(["text", "lo3"]) if n < 4 else "text", nk=nk, prec=prec, rel=rel)
        if n == 8:
            c["prec"] = "ozaki_mod"
    if c["kind"] == "adjoint":
        c.update(nk=1, rel="none", prec="fp64")
    if c["kind"] == "host":
        c["nk"] = min(c["nk"], 4) if c["cell"] == "fcc" or c["n1"] * c["n2"] * c["n3"] < 4 else 1
    return c


# ------------------------------------------------------------------ inputs
def _kpoints(c):
    """The irreducible mesh for the two-atom cell with 8 k, a shifted mesh for 27, else a
    low-discrepancy list: generic points, ragged G+k counts."""
    if c["cell"] == "fcc" and c["nk"] == 8:
        return W.FCC_IRREDUCIBLE_4x4x4
    if c["nk"] == 27:
        return W.shifted_mesh(3)
    g = 1.2207440846057596        # root of x^4 = x + 1
    i = np.arange(1, c["nk"] + 1)[:, None]
    return (0.5 + i * np.array([1 / g, 1 / g ** 2, 1 / g ** 3])) % 1.0


def _system(c, seed):
    if c["cell"] == "fcc":
        h = c["a"] / 2.0
        avec = np.array([[h, h, 0.0], [h, 0.0, h], [0.0, h, h]]).T
        sites = np.array([[0.0, 0.0, 0.0], [0.25, 0.25, 0.25]])
    else:
        n = np.array([c["n1"], c["n2"], c["n3"]])
        avec = np.diag(c["a"] * n)
        sites = np.array([(s + np.array([i, j, k])) / n for i in range(n[0]) for j in range(n[1])
                          for k in range(n[2]) for s in W.DIAMOND_CUBE_SITES])
    shift = np.random.default_rng(seed).uniform(-0.02, 0.02, size=sites.shape)
    sites = sites + shift @ np.linalg.inv(avec).T
    L, nat = c["lmax"], len(sites)
    apword = [1, 1] + [2] * (L - 1) if c["basis"] == "shipped" else [2] * (L + 1)
    lorb = {"shipped": [0, 1], "text": [0, 1, 2], "lo3": [0, 0, 0, 1, 1, 1, 2, 2, 2]}[c["basis"]]
    basis = Basis(lmaxapw=L, lmaxmat=L, apword=[apword], lorbl=[lorb], atom_species=[0] * nat)
    return W.build_system(Crystal(avec, [2.1], [0] * nat, sites.T), basis, rgkmax=c["rgkmax"], relativity=c["rel"],
                          kpoints=_kpoints(c), seed=seed)


def _states(sys, gk, seed):
    """Orthonormal columns c, weights w and energies eps of the adjoint."""
    rng = np.random.default_rng(seed + 7)
    n = sys.nmat(gk)
    z = rng.standard_normal((n, NSTATES)) + 1j * rng.standard_normal((n, NSTATES))
    return np.asfortranarray(np.linalg.qr(z)[0]), np.full(NSTATES, 2.0), rng.uniform(-0.5, 0.5, NSTATES)


def _field(seed):
    """Vector potential of a time step."""
    return np.random.default_rng(seed + 3).uniform(-5.0, 5.0, 3)


def _pmat(n, seed, device):
    """Hermitian momentum matrices of one k-point, memory [direction][column][row]."""
    g = torch.Generator(device=device).manual_seed(seed)
    x = torch.randn(3, n, n, 2, generator=g, device=device, dtype=torch.float64)
    z = torch.view_as_complex(x)
    return 0.05 * (z + z.conj().transpose(1, 2))


def _offsets(nmats):
    return [0] + list(np.cumsum([n * n for n in nmats]))


def prepare(case, seed):
    c = dict(DEFAULTS, **case)
    sys = _system(c, seed)
    gks = sys.gksets()
    ngkmax = max(g.ngp for g in gks)
    st = Setup(sys, ngkmax=ngkmax, max_batch=len(gks))
    if c["prec"] != "fp64":
        st.set_precision(c["prec"], 0)
    s = dict(kind=c["kind"], st=st, sys=sys, gks=gks, seed=seed)
    nmats = [sys.nmat(g) for g in gks]
    if c["kind"] == "host":
        s["out"] = [tuple(np.zeros((n, n), dtype=np.complex128, order="F") for _ in range(2)) for n in nmats]
        return s
    if c["kind"] == "adjoint":
        s["c"], s["w"], s["eps"] = _states(sys, gks[0], seed)
        return s
    ig = np.zeros((len(gks), ngkmax), dtype=np.int32)
    vg = np.zeros((len(gks), ngkmax, 3))
    for k, g in enumerate(gks):
        ig[k, : g.ngp], vg[k, : g.ngp] = g.igpig, g.vgpc.T
    off = _offsets(nmats)
    s["ig"], s["vg"] = torch.from_numpy(ig).cuda(), torch.from_numpy(vg).cuda()
    s["h"] = torch.empty(off[-1], dtype=torch.complex128, device="cuda")
    s["o"] = torch.empty(off[-1], dtype=torch.complex128, device="cuda")
    s["args"] = ([g.ngp for g in gks], s["ig"].data_ptr(), s["vg"].data_ptr(),
                 [s["h"].data_ptr() + 16 * int(x) for x in off[:-1]],
                 [s["o"].data_ptr() + 16 * int(x) for x in off[:-1]])
    if c["kind"] == "graph":
        s["graph"] = st.graph(*s["args"])
    if c["kind"] == "rt":
        s["p"] = [_pmat(n, seed + k, "cuda") for k, n in enumerate(nmats)]
        s["a"] = _field(seed)
    if c["kind"] == "scf":
        s["rad"] = W.mt_radial(sys, seed=seed)
        for k in ("apwfr", "lofr", "veffmt"):
            s[k] = torch.from_numpy(np.ravel(getattr(s["rad"], k), order="F").copy()).cuda()
    return s


def run(s):
    st = s["st"]
    if s["kind"] == "host":
        return st.setup_batched(s["gks"], out=s["out"])
    if s["kind"] == "adjoint":
        return st.adjoint(s["gks"][0], s["c"], s["w"], s["eps"], dveffig=True, dh=True)
    if s["kind"] == "graph":
        s["graph"].launch()
    elif s["kind"] == "rt":
        ngp, ig, vg, h, o = s["args"]
        st.rttddft_updateham_device(ngp, ig, vg, s["a"], True, [p.data_ptr() for p in s["p"]], h, o)
    else:
        if s["kind"] == "scf":
            ptrs = s["apwfr"].data_ptr(), s["lofr"].data_ptr(), s["veffmt"].data_ptr()
            st.hmlint_device(s["rad"], *ptrs)
            st.olprad_device(s["rad"], *ptrs)
            st.set_scf_inputs(keep_mt=True, keep_olp=True)
        st.setup_batched_device(*s["args"])
    return s["h"], s["o"]


# ------------------------------------------------------------------ least work
def work(case):
    c = dict(DEFAULTS, **case)
    cells = c["n1"] * c["n2"] * c["n3"]
    nat, vol = (2, c["a"] ** 3 / 4) if c["cell"] == "fcc" else (8 * cells, cells * c["a"] ** 3)
    n = vol * (c["rgkmax"] / 2.1) ** 3 / (6 * math.pi ** 2)        # plane waves in the sphere
    L = c["lmax"]
    m = 2 * (L + 1) ** 2 - (4 if c["basis"] == "shipped" else 0)   # APW rows of an atom
    lo = {"shipped": 4, "text": 9, "lo3": 27}[c["basis"]]
    dim, ngvec = n + lo * nat, vol * 12.0 ** 3 / (6 * math.pi ** 2)
    ha = 16 * nat * m * (m + lo)
    if c["kind"] == "adjoint":
        q = 4 * NSTATES
        flops = 8 * n * nat * m * q + 8 * nat * m * m * q + 16 * n * n * NSTATES / 2 + 8 * nat * m * m * NSTATES
        return {"bytes": 16 * dim * NSTATES + 2 * ha + 48 * ngvec, "flops": flops}
    flops = c["nk"] * (8 * n * n * nat * m + 8 * n * nat * m * (m + lo))
    moved = c["nk"] * 32 * dim * dim + ha + 48 * ngvec
    if c["kind"] == "rt":
        moved += c["nk"] * 48 * dim * dim
        flops += c["nk"] * 20 * dim * dim
    if c["kind"] == "scf":
        p = 2 * (L + 1) + (9 if c["basis"] == "lo3" else 3)
        moved += 8 * nat * 300 * (2 * p + 81)
        flops += 2 * nat * 84 * p * p / 2 * 300
    return {"bytes": moved, "flops": flops}


# ------------------------------------------------------------------ the same in 64 bits, plainly
def _bessel(lmax, x):
    """j_l(x), l = 0..lmax+3, by downward recurrence normalised with sum (2l+1) j_l^2 = 1."""
    top = lmax + 60
    x = np.maximum(x, 1e-30)
    j = np.zeros((top + 2, x.size))
    j[top] = 1.0
    for l in range(top, 0, -1):
        j[l - 1] = (2 * l + 1) / x * j[l] - j[l + 1]
        j[:, np.abs(j[l - 1]) > 1e100] *= 1e-100
    return (j / np.sqrt(((2 * np.arange(top + 2) + 1)[:, None] * j ** 2).sum(axis=0)))[: lmax + 4]


def _derivatives(j, m):
    """m-th derivatives of j_l, l = 0..len-1-m, by j_l' = (l j_{l-1} - (l+1) j_{l+1}) / (2l+1)."""
    for _ in range(m):
        n = j.shape[0] - 1
        l = np.arange(n)[:, None]
        below = np.concatenate([np.zeros((1, j.shape[1])), j[: n - 1]])
        j = (l * below - (l + 1) * j[1: n + 1]) / (2 * l + 1)
    return j


def _ylm(lmax, v):
    """Y_lm of the directions v (3, n): array ((lmax+1)^2, n), rows l(l+1)+m."""
    r = np.sqrt((v * v).sum(axis=0))
    ct = np.where(r > 1e-14, v[2] / np.maximum(r, 1e-300), 1.0)
    st = np.sqrt(np.maximum(0.0, (v[0] ** 2 + v[1] ** 2))) / np.maximum(r, 1e-300)
    ph = np.where(np.hypot(v[0], v[1]) > 1e-14, np.arctan2(v[1], v[0]), 0.0)
    y = np.zeros(((lmax + 1) ** 2, v.shape[1]), dtype=np.complex128)
    d = np.full(v.shape[1], 1.0 / math.sqrt(4 * math.pi))
    for m in range(lmax + 1):
        if m:
            d = -math.sqrt((2 * m + 1) / (2.0 * m)) * st * d
        p0, p1, a0 = np.zeros_like(d), d, 1.0
        for l in range(m, lmax + 1):
            if l > m:
                a = math.sqrt((4.0 * l * l - 1) / (l * l - m * m))
                p0, p1, a0 = p1, a * (ct * p1 - p0 / a0), a
            y[l * (l + 1) + m] = p1 * np.exp(1j * m * ph)
            y[l * (l + 1) - m] = (-1) ** m * np.conj(y[l * (l + 1) + m])
    return y


def _rows(basis):
    """(l, lm, io) of the APW rows and (l, lm, ilo) of the local-orbital rows of an atom."""
    apw = [(l, l * (l + 1) + m, io) for l in range(basis.lmaxmat + 1) for m in range(-l, l + 1)
           for io in range(basis.apword[0][l])]
    lo = [(l, l * (l + 1) + m, i) for i, l in enumerate(basis.lorbl[0]) for m in range(-l, l + 1)]
    return apw, lo


def _match(sys, gk, dev):
    """Matching coefficients (APW rows, ngp) of each atom in turn."""
    b, cr = sys.basis, sys.crystal
    L, R = b.lmaxmat, sys.rmt[0]
    v = np.asarray(gk.vgpc)
    g = np.sqrt((v * v).sum(axis=0))
    omax = max(b.apword[0])
    j = _bessel(L, g * R)
    dj = np.stack([_derivatives(j, i)[: L + 1] * g ** i for i in range(omax)])
    y = _ylm(L, v).conj() * (4 * math.pi / math.sqrt(cr.omega))
    r = sys.spr_tail[:, 0]
    t = (r - R) / (r[-1] - r[0])                                    # scaled distances from the sphere
    inv = np.linalg.inv(np.vander(t, len(t), increasing=True))
    yt, vt = torch.from_numpy(y).to(dev), torch.from_numpy(v).to(dev)
    djt = torch.from_numpy(dj).to(dev)
    apw, _ = _rows(b)
    lm = torch.tensor([x[1] for x in apw], device=dev)
    for ias in range(sys.natmtot):
        radial = {}
        for l in range(L + 1):
            n = b.apword[0][l]
            poly = inv @ sys.apwfr_tail[:, :n, l, ias]              # u = sum_k poly_k t^k
            d = np.array([[math.factorial(i) * poly[i, o] / (r[-1] - r[0]) ** i for o in range(n)] for i in range(n)])
            sol = torch.from_numpy(np.linalg.inv(d)).to(dev) @ djt[:n, l]
            for io in range(n):
                radial[l, io] = sol[io] * (1j ** l)
        coef = torch.stack([radial[l, io] for l, _, io in apw]) * yt[lm]
        tau = torch.from_numpy(np.asarray(cr.atposc[:, ias])).to(dev)
        yield coef * torch.exp(1j * (tau @ vt))


def _box(sys, gk, dev):
    """Index of every G_i - G_j in the G list: (ngp, ngp), and the validity mask."""
    gv = sys.gv
    iv = torch.from_numpy(np.asarray(gv.ivg)[:, np.asarray(gk.igpig) - 1].astype(np.int64)).to(dev)
    lo, box = np.asarray(gv.intgv)[:, 0], torch.from_numpy(np.asarray(gv.ivgig).astype(np.int64)).to(dev)
    d = [iv[x][:, None] - iv[x][None, :] - int(lo[x]) for x in range(3)]
    ig = box[d[0], d[1], d[2]]
    return (ig - 1).clamp(min=0), (ig >= 1) & (ig <= gv.ngvec)


def _h1(sys):
    return sys.relativity == "iora*"


def _hamiltonian(sys, gk, dev):
    """H and O of one k-point, (row, column)."""
    b, n = sys.basis, gk.ngp
    apw, lo = _rows(b)
    nlo, dim = len(lo), sys.nmat(gk)
    H = torch.zeros(dim, dim, dtype=torch.complex128, device=dev)
    O = torch.zeros(dim, dim, dtype=torch.complex128, device=dev)
    up = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(dev)  # noqa: E731
    for ias, A in enumerate(_match(sys, gk, dev)):
        m = A.shape[0]
        h, C = up(sys.mt_aa[:m, :m, ias]), A
        if _h1(sys):
            w = torch.zeros(m, m, dtype=torch.complex128, device=dev)
            for f, (_, lmf, io) in enumerate(apw):
                for q, (_, lmq, jo) in enumerate(apw):
                    if lmf == lmq:
                        w[q, f] = float(sys.h1aa[io, jo, apw[f][0], ias])
            C = A + w @ A
        H[:n, :n] += A.conj().T @ (h @ A)
        O[:n, :n] += A.conj().T @ C
        if not nlo:
            continue
        s = slice(n + ias * nlo, n + (ias + 1) * nlo)
        H[s, :n] = up(sys.mt_loa[:nlo, :m, ias]) @ A
        H[:n, s] = H[s, :n].conj().T
        hl = up(sys.mt_lolo[:nlo, :nlo, ias])
        H[s, s] = hl.triu() + hl.triu(1).conj().T
        S = np.zeros((nlo, m))
        D = np.zeros((nlo, nlo))
        for r, (_, lmr, i) in enumerate(lo):
            for f, (_, lmf, io) in enumerate(apw):
                if lmr == lmf:
                    S[r, f] = sys.oalo[io, i, ias] + (sys.h1loa[io, i, ias] if _h1(sys) else 0.0)
            for q, (_, lmq, i2) in enumerate(lo):
                if lmr == lmq:
                    x, z = (i, i2) if r <= q else (i2, i)
                    D[r, q] = sys.ololo[x, z, ias] + (sys.h1lolo[x, z, ias] if _h1(sys) else 0.0)
        O[s, :n] = up(S).to(torch.complex128) @ A
        O[:n, s] = O[s, :n].conj().T
        O[s, s] = up(D).to(torch.complex128)
    ig, ok = _box(sys, gk, dev)
    v = up(gk.vgpc)
    half = 0.5 * (v.T @ v) * ok
    ngv = sys.gv.ngvec
    H[:n, :n] += up(sys.veffig[:ngv])[ig] * ok + up(sys.kinetic_weight[:ngv])[ig] * half
    O[:n, :n] += up(sys.cfunig[:ngv])[ig] * ok
    if _h1(sys):
        O[:n, :n] += up(sys.m2effig[:ngv])[ig] * half * (0.5 / 137.03599911 ** 2)
    for M in (H, O):      # upper triangle and its conjugate
        M[:n, :n] = M[:n, :n].triu() + M[:n, :n].triu(1).conj().T
    return H, O


def _spline_weights(x):
    """w with sum w f = integral of the cubic spline through (x, f) whose end second derivatives are
    the second divided differences of the three points at either end."""
    n = len(x)
    h = np.diff(x)
    slope = np.zeros((n - 1, n))
    for i in range(n - 1):
        slope[i, i], slope[i, i + 1] = -1 / h[i], 1 / h[i]
    M, rhs = np.zeros((n, n)), np.zeros((n, n))
    M[0, 0] = M[-1, -1] = 1.0
    rhs[0] = (slope[1] - slope[0]) / (x[2] - x[0])
    rhs[-1] = (slope[-1] - slope[-2]) / (x[-1] - x[-3])
    for i in range(1, n - 1):
        M[i, i - 1], M[i, i], M[i, i + 1] = h[i - 1], 2 * (h[i - 1] + h[i]), h[i]
        rhs[i] = 3 * (slope[i] - slope[i - 1])
    c = np.linalg.solve(M, rhs)
    w = np.zeros(n)
    for i in range(n - 1):
        d = (c[i + 1] - c[i]) / (3 * h[i])
        b = slope[i] - (c[i] + d * h[i]) * h[i]
        w += h[i] ** 4 / 4 * d + h[i] ** 3 / 3 * c[i] + h[i] ** 2 / 2 * b
        w[i] += h[i]
    return w


@functools.lru_cache(maxsize=4)
def _gaunt(lmax, lmaxvr):
    """Integrals of conj(Y_1) R_2 Y_3 (R real harmonics) by quadrature, [lm1][lm3][lm2]."""
    nt, nf = lmax + lmaxvr // 2 + 2, 2 * lmax + lmaxvr + 2
    z, wz = np.polynomial.legendre.leggauss(nt)
    f = 2 * math.pi * np.arange(nf) / nf
    z, f = np.repeat(z, nf), np.tile(f, nt)
    w = np.repeat(wz, nf) * 2 * math.pi / nf
    s = np.sqrt(1 - z * z)
    v = np.stack([s * np.cos(f), s * np.sin(f), z])
    y, y2 = _ylm(lmax, v), _ylm(lmaxvr, v)
    r2 = np.zeros(y2.shape)
    for l in range(lmaxvr + 1):
        for m in range(-l, l + 1):
            t = y2[l * (l + 1) + m]
            r2[l * (l + 1) + m] = t.real if m == 0 else math.sqrt(2) * (t.real if m > 0 else t.imag)
    y, r2 = torch.from_numpy(y), torch.from_numpy(r2 * w).to(torch.complex128)
    prod = (y.conj()[:, None, :] * y[None, :, :]).reshape(-1, y.shape[1])
    return (prod @ r2.T).reshape(y.shape[0], y.shape[0], -1)


def _integrals(sys, rad):
    """mt_aa, mt_loa, mt_lolo, oalo, ololo of the radial functions and potential, put into sys."""
    b = sys.basis
    apw, lo = _rows(b)
    gnt = _gaunt(b.lmaxmat, rad.lmaxvr)
    nr = int(rad.nrmt[0])
    r = rad.spr[:nr, 0]
    w = _spline_weights(r)
    funs = [(l, io) for l in range(b.lmaxmat + 1) for io in range(b.apword[0][l])]
    nrad = len(funs)
    row = [(lm, funs.index((l, io))) for l, lm, io in apw] + [(lm, nrad + i) for _, lm, i in lo]
    ls = np.array([l for l, _ in funs] + list(b.lorbl[0]))
    lm, pf = torch.tensor([x[0] for x in row]), torch.tensor([x[1] for x in row])
    same = (lm[:, None] == lm[None, :])
    g = gnt[lm[:, None], lm[None, :]]
    na, nl = len(apw), len(lo)
    for ias in range(sys.natmtot):
        u = np.stack([rad.apwfr[:nr, 0, io, l, ias] for l, io in funs] + [rad.lofr[:nr, 0, i, ias] for i in range(len(b.lorbl[0]))])
        d = np.stack([rad.apwfr[:nr, 1, io, l, ias] for l, io in funs] + [rad.lofr[:nr, 1, i, ias] for i in range(len(b.lorbl[0]))])
        pot = rad.veffmt[:, :nr, ias]
        a = 0.5 / 137.03599911 ** 2 if sys.relativity != "none" else 0.0
        rm = 1 / (1 - a * pot[0] * W.Y00)
        I = torch.from_numpy(np.einsum("pr,qr,vr->pqv", u, u * (w * r * r), pot, optimize=True))
        kin = lambda f: 0.5 * ((d * (f * r * r)) @ d.T + (ls * (ls + 1))[None, :] * ((u * f) @ u.T))  # noqa: E731
        z = (g * I[pf[:, None], pf[None, :]]).sum(-1) + same * torch.from_numpy(kin(w * rm))[pf[:, None], pf[None, :]]
        z = z.numpy()
        sys.mt_aa[:na, :na, ias], sys.mt_loa[:nl, :na, ias], sys.mt_lolo[:nl, :nl, ias] = z[:na, :na], z[na:, :na], z[na:, na:]
        ov, h1 = (u * (w * r * r)) @ u.T, kin(w * a * rm * rm)
        for i, l in enumerate(b.lorbl[0]):
            for io in range(b.apword[0][l]):
                p = funs.index((l, io))
                sys.oalo[io, i, ias] = ov[p, nrad + i]
                if _h1(sys):
                    sys.h1loa[io, i, ias] = h1[p, nrad + i]
            for i2, l2 in enumerate(b.lorbl[0]):
                sys.ololo[i, i2, ias] = ov[nrad + i, nrad + i2] if l == l2 else 0.0
                if _h1(sys):
                    sys.h1lolo[i, i2, ias] = h1[nrad + i, nrad + i2] if l == l2 else 0.0
        if _h1(sys):
            for l in range(b.lmaxmat + 1):
                n = b.apword[0][l]
                p = funs.index((l, 0))
                sys.h1aa[:n, :n, l, ias] = h1[p: p + n, p: p + n]


def _gradients(sys, gk, c, w, eps, dev):
    """dL/dtau, dL/dV and dL/dh of L = sum_n w_n c_n^H (H - eps_n O) c_n."""
    b, n, cr = sys.basis, gk.ngp, sys.crystal
    apw, lo = _rows(b)
    m, nlo, nat = len(apw), len(lo), sys.natmtot
    up = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(dev)  # noqa: E731
    c, w, eps, v = up(c), up(w), up(eps), up(gk.vgpc)
    cg = c[:n]
    ig, ok = _box(sys, gk, dev)
    ngv = sys.gv.ngvec
    P, Q = (cg.conj() * w) @ cg.T, (cg.conj() * (w * eps)) @ cg.T
    scatter = lambda x: torch.zeros(ngv, dtype=torch.complex128, device=dev).index_put_((ig[ok],), x[ok], accumulate=True)  # noqa: E731
    dv = scatter(P)
    R = scatter(P * (0.5 * (v.T @ v)) - Q)
    gvec = up(np.asarray(sys.gv.vgc)[:, :ngv])
    gl = gvec.norm(dim=0)
    x = gl * sys.rmt[0]
    ff = torch.where(gl > 1e-6, 4 * math.pi / cr.omega * (torch.sin(x) - x * torch.cos(x)) / gl.clamp(min=1e-6) ** 3,
                     torch.full_like(gl, 4 * math.pi / (3 * cr.omega) * sys.rmt[0] ** 3))
    dtau = np.zeros((3, nat))
    dh = np.zeros((b.maxaa, b.maxaa, nat), dtype=np.complex128)
    for ias, A in enumerate(_match(sys, gk, dev)):
        U = A @ cg
        h = up(sys.mt_aa[:m, :m, ias])
        dh[:m, :m, ias] = ((U.conj() * w) @ U.T).cpu().numpy()
        left = h @ U - U * eps
        if nlo:
            S = np.zeros((nlo, m))
            for r, (_, lmr, i) in enumerate(lo):
                for f, (_, lmf, io) in enumerate(apw):
                    if lmr == lmf:
                        S[r, f] = sys.oalo[io, i, ias]
            cl = c[n + ias * nlo: n + (ias + 1) * nlo]
            loa, S = up(sys.mt_loa[:nlo, :m, ias]), up(S).to(torch.complex128)
            left = left + loa.conj().T @ cl - S.T @ cl * eps
        tau = up(np.asarray(cr.atposc[:, ias]))
        phase = ff * torch.exp(-1j * (tau @ gvec)) * R
        for d in range(3):
            Ud = 1j * (A @ (v[d][:, None] * cg))
            t = 2 * (w * (left.conj() * Ud).sum(0)).sum().real + (1j * gvec[d] * phase).sum().real
            dtau[d, ias] = float(t)
    return dtau, dv.cpu().numpy(), dh


def exact(case, seed):
    c = dict(DEFAULTS, **case)
    sys = _system(c, seed)
    gks = sys.gksets()
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if c["kind"] == "adjoint":
        return _gradients(sys, gks[0], *_states(sys, gks[0], seed), dev)
    if c["kind"] == "scf":
        _integrals(sys, W.mt_radial(sys, seed=seed))
    both = [_hamiltonian(sys, g, dev) for g in gks]
    if c["kind"] == "host":
        return [(H.cpu().numpy(), O.cpu().numpy()) for H, O in both]
    if c["kind"] == "rt":
        a, light = _field(seed), 299792458.0 * 2.418884326509e-17 / 0.52917721067e-10     # c in atomic units
        out = []
        for k, (H, O) in enumerate(both):
            p = _pmat(H.shape[0], seed + k, dev)
            H = H + float(a @ a) / (2 * light ** 2) * O + sum(float(a[i]) / light * p[i].T for i in range(3))
            out.append((H, O))
        both = out
    return tuple(torch.cat([M[q].T.reshape(-1) for M in both]) for q in range(2))
