"""The modular products where their form changes: contraction lengths on both sides of 8192 (256 x 128
tiles with the short residue reduction, 256 x 256 tiles), the paced launches of large cells, and batches whose
residues are formed in more than one chunk.
"""
import numpy as np
import pytest

import lapw_oracle as O
from exciting_b200 import workloads as W
from exciting_b200.basis import Basis
from exciting_b200.crystal import Crystal, GkSet

pytestmark = pytest.mark.gpu

TOL_FRO = 1e-12
SIZES = [1, 17, 64, 127, 128, 129, 255, 256, 257, 385]


def _cell(nat, a, *, lmax=8, rgkmax=10.0, relativity="none", nk=1):
    h = a / 2.0
    avec = np.array([[h, h, 0.0], [h, 0.0, h], [0.0, h, h]]).T
    rng = np.random.default_rng(nat)
    b = Basis(lmaxapw=lmax, lmaxmat=lmax, apword=[[1] * (lmax + 1)], lorbl=[[0, 1]], atom_species=[0] * nat)
    return W.build_system(Crystal(avec, [2.1], [0] * nat, rng.uniform(size=(3, nat))), b, rgkmax=rgkmax,
                          relativity=relativity, kpoints=rng.uniform(size=(nk, 3)), seed=nat)


def _shortest(g, n):
    i = np.argsort(g.gpc, kind="stable")[:n]
    return GkSet(vpl=g.vpl, ngp=len(i), igpig=np.ascontiguousarray(g.igpig[i]),
                 vgpc=np.ascontiguousarray(g.vgpc[:, i]), gpc=g.gpc[i], tpgpc=np.ascontiguousarray(g.tpgpc[:, i]))


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def _outputs(st, gks):
    import torch
    return [[torch.empty(2 * (g.ngp + st.nlotot) ** 2, dtype=torch.float64, device="cuda") for _ in range(2)]
            for g in gks]


def _run(st, gks, out=None):
    """H and O of every k-point in one call, as device tensors."""
    import torch
    ig = np.zeros((len(gks), st.ngkmax), dtype=np.int32)
    vg = np.zeros((len(gks), st.ngkmax, 3))
    for k, g in enumerate(gks):
        ig[k, : g.ngp] = g.igpig
        vg[k, : g.ngp] = g.vgpc.T
    ig, vg = torch.from_numpy(ig).cuda(), torch.from_numpy(vg).cuda()
    out = out or _outputs(st, gks)
    for pair in out:
        for z in pair:
            z.fill_(float("nan"))
    torch.cuda.synchronize()
    st.setup_batched_device([g.ngp for g in gks], ig.data_ptr(), vg.data_ptr(), [h.data_ptr() for h, _ in out],
                            [o.data_ptr() for _, o in out])
    st.synchronize()
    return out


def _same(x, y):
    import torch
    return all(torch.equal(a, b) for a, b in zip(x, y))


@pytest.mark.parametrize("relativity", ["none", "iora*"])
@pytest.mark.parametrize("nat", [101, 102])                     # K = 8181 and 8262
def test_tile_edges_beside_the_change_of_form(nat, relativity):
    from exciting_b200.fvsystem import Setup
    s = _cell(nat, 10.26, relativity=relativity)
    full = s.gkset(s.kpoints[0])
    assert full.ngp >= SIZES[-1]
    gks = [_shortest(full, n) for n in SIZES]
    st = Setup(s, ngkmax=SIZES[-1], max_batch=len(SIZES))
    st.set_precision("ozaki_mod", 0)
    batch = st.setup_batched(gks)
    for g, (h, o) in zip(gks, batch):
        hr, orf = O.hamiltonandoverlapsetup(s, g)
        assert _rel(h, hr) <= TOL_FRO and _rel(o, orf) <= TOL_FRO, (g.ngp, _rel(h, hr), _rel(o, orf))
        off = ~np.eye(h.shape[0], dtype=bool)
        assert np.array_equal(h[off], h.conj().T[off]) and np.array_equal(o[off], o.conj().T[off]), g.ngp
        h1, o1 = st.setup_batched([g])[0]
        assert np.array_equal(h, h1) and np.array_equal(o, o1), g.ngp
    st.close()


@pytest.mark.parametrize("nat", [101, 102])
def test_paced_launches(nat):
    """Operand planes of one product above 100 MB: the clusters of a launch pace each other."""
    import torch
    from exciting_b200.fvsystem import Setup
    s = _cell(nat, 17.0, rgkmax=12.5)
    g = _shortest(s.gkset(s.kpoints[0]), 4321)
    assert g.ngp == 4321
    st = Setup(s, ngkmax=g.ngp)
    (h64, o64), = _run(st, [g])
    st.set_precision("ozaki_mod", 0)
    first = _run(st, [g])[0]
    for x, y in zip(first, (h64, o64)):
        assert float(torch.linalg.norm(x - y)) <= TOL_FRO * float(torch.linalg.norm(y))
    assert _same(first, _run(st, [g])[0])
    st.close()


def test_per_atom_products_in_two_chunks():
    """Ten k-points of 101 atoms: 1010 tiles of 0.64 MB of residues in a buffer of 512 MB."""
    from exciting_b200.fvsystem import Setup
    s = _cell(101, 10.26, nk=10)
    gks = [_shortest(s.gkset(v), 200 - 3 * i) for i, v in enumerate(s.kpoints)]
    st = Setup(s, ngkmax=200, max_batch=len(gks))
    st.set_precision("ozaki_mod", 0)
    batch = _run(st, gks)
    st.close()
    one = Setup(s, ngkmax=200)
    one.set_precision("ozaki_mod", 0)
    for g, x in zip(gks, batch):
        assert _same(x, _run(one, [g])[0]), g.ngp
    one.close()


def test_hamiltonian_products_in_chunks():
    """40 k-points of about 1900 G+k: 4.7 GB of H and O residues, in chunks of at most 4 GB, then, with little
    device memory left, in more and smaller ones."""
    import torch
    from exciting_b200.fvsystem import Setup
    s = _cell(2, 13.2, rgkmax=12.5, nk=40)
    gks = [_shortest(s.gkset(v), 2000 - 7 * i) for i, v in enumerate(s.kpoints)]
    assert gks[0].ngp == 2000
    tiles = sum(1 for g in gks for ib in range((g.ngp + 255) // 256) for jb in range((g.ngp + 127) // 128)
                if jb * 128 + 127 >= ib * 256)
    assert tiles * 28 * 256 * 256 > 4 << 30
    one = Setup(s, ngkmax=2000)
    one.set_precision("ozaki_mod", 0)
    alone = [_run(one, [g])[0] for g in gks]
    one.close()
    st = Setup(s, ngkmax=2000, max_batch=len(gks))
    st.set_precision("ozaki_mod", 0)
    out = _outputs(st, gks)
    assert all(_same(x, y) for x, y in zip(alone, _run(st, gks, out)))
    st.set_precision("ozaki", 7)                                # 0.6 GB of operands in place of 1.2 GB, no residues
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (4 << 30), dtype=torch.uint8, device="cuda")
    st.set_precision("ozaki_mod", 0)
    left = torch.cuda.mem_get_info()[0]
    assert all(_same(x, y) for x, y in zip(alone, _run(st, gks, out)))
    del hog
    st.close()
    torch.cuda.empty_cache()
    assert left < 2 << 30                                       # the full buffer had not fitted: half of it was taken
