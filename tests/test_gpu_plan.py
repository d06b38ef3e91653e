"""Launch plans of the thread kernels (several lanes to a quartet in the buckets that would
outlast the launch): J, K and the counted quartets against the oracle from lists of a few
entries, where every heavy bucket is split over a whole warp, to lists with split and
unsplit buckets side by side; bitwise equal however a deterministic build is launched."""

import numpy as np
import pytest

from tonto_b200.molecules import water_cluster

TOL = 1e-11          # the element bar of every FP64 build


def _density(mol, seed):
    A = np.random.default_rng(seed).normal(size=(mol.n_bf, mol.n_bf)) * 0.03
    return A + A.T


@pytest.mark.gpu
@pytest.mark.parametrize("n,basis", [(1, "STO-3G"), (1, "cc-pVDZ"), (2, "6-31G(d)"), (5, "cc-pVDZ")])
def test_split_quartets_match_the_oracle(cuda_ok, oracle_mod, n, basis):
    from tonto_b200.fock import TF_JK_MIXED, FockBuilder
    mol = water_cluster(n, seed=40 + n, basis=basis)
    P = _density(mol, n)
    orc = oracle_mod.Oracle(mol, schwarz_cutoff=1e-12)
    orc.counts(reset=True)
    Jr, Kr = orc.jk(P)
    cnt = orc.counts(reset=True).reshape(625, 2)
    fb = FockBuilder(mol, schwarz_cutoff=1e-12)
    for v in range(4):
        fb.set_kernel_variant(v)
        for _ in range(2):
            J, K = fb.make_r_JK(P)
            assert np.max(np.abs(J - Jr)) <= TOL and np.max(np.abs(K - Kr)) <= TOL
            st = fb.stats()
            assert (st["quartets"], st["prim_quartets"]) == (cnt[:, 0].sum(), cnt[:, 1].sum())
    J, K = fb.make_r_JK(P, TF_JK_MIXED)
    assert np.max(np.abs(J - Jr)) <= 1e-9 and np.max(np.abs(K - Kr)) <= 1e-9
    fb.close()
    fd = FockBuilder(mol, schwarz_cutoff=1e-12, deterministic=True)
    a, b = fd.make_r_JK(P), fd.make_r_JK(P)          # class launches, then a replayed graph
    fd.set_graph(False)
    fd.set_list_budget(1 << 10)                      # one class pair a chunk
    c = fd.make_r_JK(P)
    fd.close()
    for x, y, z in zip(a, b, c):
        assert np.array_equal(x, y) and np.array_equal(x, z)
