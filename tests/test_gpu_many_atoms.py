"""iora* with more (atom, l) pairs than a grid's y extent (65,535)."""
import numpy as np
import pytest

import lapw_oracle as O
from exciting_b200 import workloads as W
from exciting_b200.basis import Basis
from exciting_b200.crystal import Crystal, GkSet

pytestmark = pytest.mark.gpu


def test_iora_overlap_of_33000_atoms():
    from exciting_b200.fvsystem import Setup
    nat = 33000
    h = 5.13
    avec = np.array([[h, h, 0.0], [h, 0.0, h], [0.0, h, h]]).T
    b = Basis(lmaxapw=1, lmaxmat=1, apword=[[1, 1]], lorbl=[[]], atom_species=[0] * nat)
    s = W.build_system(Crystal(avec, [2.1], [0] * nat, np.random.default_rng(5).uniform(size=(3, nat))), b, rgkmax=4.0,
                       gmaxvr=4.0, relativity="iora*", kpoints=np.array([[0.13, 0.37, 0.21]]), seed=5)
    g = s.gkset(s.kpoints[0])
    n = min(g.ngp, 12)
    g = GkSet(vpl=g.vpl, ngp=n, igpig=np.ascontiguousarray(g.igpig[:n]), vgpc=np.ascontiguousarray(g.vgpc[:, :n]),
              gpc=g.gpc[:n], tpgpc=np.ascontiguousarray(g.tpgpc[:, :n]))
    st = Setup(s, ngkmax=n)
    st.set_precision("fp64")
    hd, od = st.setup_batched([g])[0]
    hr, orf = O.hamiltonandoverlapsetup(s, g)
    assert np.linalg.norm(hd - hr) <= 1e-12 * np.linalg.norm(hr)
    assert np.linalg.norm(od - orf) <= 1e-12 * np.linalg.norm(orf)
    st.close()
