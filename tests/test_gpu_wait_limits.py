"""Waits of the tensor-core pipelines that run out anywhere in a product, without a GPU fault.

The wait limit (exs_set_wait_limit) is lowered to lengths between one cycle and longer than a whole
kernel, so that producers, the MMA issuer and the epilogues give up at different points: before the first
copy has landed, with MMAs under way, between the two accumulators of the 256-column tiles.  Every call
either reports EXS_ERR_TIMEOUT or returns the same bits as without a limit, and the context goes on with
the same bits once the limit is taken away.
"""
import numpy as np
import pytest

from exciting_b200 import workloads as W
from exciting_b200.abi import ExsError
from exciting_b200.basis import Basis
from exciting_b200.crystal import Crystal

pytestmark = pytest.mark.gpu

EXS_ERR_TIMEOUT = -7
LIMITS = [1, 150, 400, 700, 1000, 1500, 2500, 5000, 10000, 30000, 100000]


def _cell(name):
    if name == "two_atoms":
        return W.si_fcc("text")
    nat = 102                                              # K = 8262: the products' 256 x 256 tiles
    pos = np.random.default_rng(3).uniform(size=(3, nat))
    b = Basis(lmaxapw=8, lmaxmat=8, apword=[[1] * 9], lorbl=[[0]], atom_species=[0] * nat)
    h = 5.13
    avec = np.array([[h, h, 0.0], [h, 0.0, h], [0.0, h, h]]).T
    return W.build_system(Crystal(avec, [2.1], [0] * nat, pos), b, rgkmax=10.0,
                          kpoints=np.array([[0.13, 0.37, 0.21]]), seed=7)


@pytest.mark.parametrize("cell,mode,count,config", [("two_atoms", "ozaki_mod", 0, 0), ("long", "ozaki_mod", 0, 0),
                                                    ("two_atoms", "ozaki", 7, 0), ("two_atoms", "ozaki", 7, 7),
                                                    ("two_atoms", "ozaki", 7, 8), ("two_atoms", "ozaki", 7, 9)])
def test_short_waits_report_or_finish(cell, mode, count, config):
    from exciting_b200.fvsystem import Setup
    s = _cell(cell)
    gks = [s.gkset(v) for v in s.kpoints[:3]]
    st = Setup(s, max_batch=len(gks))
    st.set_precision(mode, count)
    st.set_kernel_config(config)

    def same(got):
        return all(np.array_equal(a, b) for x, y in zip(got, ref) for a, b in zip(x, y))

    ref = st.setup_batched(gks)
    ran_out = []
    for limit in LIMITS:
        st.set_wait_limit(limit)
        try:
            got = st.setup_batched(gks)
        except ExsError as e:
            assert e.code == EXS_ERR_TIMEOUT
            ran_out.append(limit)
        else:
            assert same(got), limit
    assert LIMITS[0] in ran_out
    st.set_wait_limit(0)
    assert same(st.setup_batched(gks))
    st.close()
