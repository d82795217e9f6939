"""H and O where the tiles of the device kernels end: G+k counts on both sides of the 16, 32, 64, 128 and
256 edges, odd contraction lengths, per-atom blocks of one and of two row groups, and the layouts of the
matching coefficients (1 to 3 APW orders, species of unequal bases, lmaxmat below lmaxapw, no local orbitals).

Both precisions are held to the metric's bar against the FP64 oracle; with three APW orders, whose
coefficients hang on second derivatives at the sphere, to ten times what one unit in the last place of the
radial functions does to the oracle's own H and O.  H is Hermitian bit for bit, and a
k-point has the same bits alone, where the FP64 products take their smallest tiles, as in a batch.
"""
import copy

import numpy as np
import pytest

import lapw_oracle as O
from exciting_b200 import workloads as W
from exciting_b200.basis import Basis
from exciting_b200.crystal import Crystal, GkSet

pytestmark = pytest.mark.gpu

TOL_FRO = 1e-12
SIZES = [1, 2, 15, 16, 17, 31, 33, 64, 65, 127, 128, 129, 255, 256, 257, 385]


def _cell(name):
    h = 5.13
    avec = np.array([[h, h, 0.0], [h, 0.0, h], [0.0, h, h]]).T
    pos = np.array([[0.01, -0.02, 0.015], [0.25, 0.26, 0.24]]).T
    kw = dict(rgkmax=10.0, kpoints=np.array([[0.13, 0.37, 0.21]]), seed=11)
    if name in ("none", "zora", "iora*"):                       # K = 2 * 162
        b = Basis(lmaxapw=8, lmaxmat=8, apword=[[2] * 9], lorbl=[[0, 1, 2]], atom_species=[0, 0])
        return W.build_system(Crystal(avec, [2.1], [0, 0], pos), b, relativity=name, **kw)
    if name == "two_row_blocks":                                # 242 APW rows + 27 local orbitals per atom
        b = Basis(lmaxapw=10, lmaxmat=10, apword=[[2] * 11], lorbl=[[0] * 3 + [1] * 3 + [2] * 3],
                  atom_species=[0, 0])
        return W.build_system(Crystal(avec, [2.1], [0, 0], pos), b, **kw)
    if name.startswith("orders_1_to_3"):                             # unequal species, odd K, one without local orbitals
        b = Basis(lmaxapw=7, lmaxmat=5, apword=[[3, 2, 1, 1, 2, 3, 1, 1], [1, 3, 2, 2, 1, 1, 2, 2]],
                  lorbl=[[], [2, 0, 1]], atom_species=[0, 1])
        return W.build_system(Crystal(avec, [2.1, 1.9], [0, 1], pos), b,
                              relativity="iora*" if name.endswith("iora*") else "none", **dict(kw, rgkmax=8.5))
    if name == "no_lo":
        b = Basis(lmaxapw=3, lmaxmat=3, apword=[[1] * 4], lorbl=[[]], atom_species=[0, 0])
        return W.build_system(Crystal(avec, [2.1], [0, 0], pos), b, **kw)
    raise ValueError(name)


def _gksets(s):
    """The k-point's G+k vectors in order of length, cut at each of SIZES."""
    g = s.gkset(s.kpoints[0])
    order = np.argsort(g.gpc, kind="stable")
    assert g.ngp >= SIZES[-1], g.ngp
    cut = [order[:n] for n in SIZES]
    return [GkSet(vpl=g.vpl, ngp=len(i), igpig=np.ascontiguousarray(g.igpig[i]),
                  vgpc=np.ascontiguousarray(g.vgpc[:, i]), gpc=g.gpc[i], tpgpc=np.ascontiguousarray(g.tpgpc[:, i]))
            for i in cut]


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def _tolerance(s, g):
    t = copy.copy(s)
    ulp = np.finfo(float).eps * np.random.default_rng(0).choice([-1, 0, 1], size=s.apwfr_tail.shape)
    t.apwfr_tail = np.asfortranarray(s.apwfr_tail * (1 + ulp))
    pairs = zip(O.hamiltonandoverlapsetup(t, g), O.hamiltonandoverlapsetup(s, g))
    return max(TOL_FRO, 10 * max(_rel(a, b) for a, b in pairs))


@pytest.mark.parametrize("prec", ["fp64", "ozaki_mod"])
@pytest.mark.parametrize("cell", ["none", "zora", "iora*", "two_row_blocks", "orders_1_to_3",
                                  "orders_1_to_3 iora*", "no_lo"])
def test_tile_edges(cell, prec):
    from exciting_b200.fvsystem import Setup
    s = _cell(cell)
    gks = _gksets(s)
    st = Setup(s, ngkmax=SIZES[-1], max_batch=len(SIZES))
    st.set_precision(prec, 0)                                # 0: the full set of moduli
    batch = st.setup_batched(gks)
    tol = _tolerance(s, gks[-1]) if s.basis.apwordmax > 2 else TOL_FRO
    for g, (h, o) in zip(gks, batch):
        hr, orf = O.hamiltonandoverlapsetup(s, g)
        assert _rel(h, hr) <= tol, (g.ngp, _rel(h, hr))
        assert _rel(o, orf) <= tol, (g.ngp, _rel(o, orf))
        off = ~np.eye(h.shape[0], dtype=bool)
        assert np.array_equal(h[off], h.conj().T[off]), g.ngp
        assert np.array_equal(o[off], o.conj().T[off]), g.ngp
        h1, o1 = st.setup_batched([g])[0]
        assert np.array_equal(h, h1) and np.array_equal(o, o1), g.ngp
    # coefficients that the caller supplies, in the reference's layout
    for g, (h, o) in list(zip(gks, batch))[-3:]:
        apwalm, _ = st.match(g)
        h2, o2 = st.hamiltonandoverlapsetup(g, apwalm)
        assert _rel(h2, h) <= TOL_FRO and _rel(o2, o) <= TOL_FRO, g.ngp
