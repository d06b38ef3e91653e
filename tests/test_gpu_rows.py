"""The lane-group kernels (pp, dp, dd and f shells) against the oracle where they can go
wrong: lists shorter than a warp's groups and not a multiple of them (one molecule), every
ket width up to (ff| (two and three warps a quartet), Cartesian and spherical, restricted
and unrestricted rows, J or K alone."""

import numpy as np
import pytest

from tonto_b200.molecules import water_cluster

TOL = 1e-11          # the element bar of every FP64 build; densities of order 0.1


def _density(mol, seed):
    A = np.random.default_rng(seed).normal(size=(mol.n_bf, mol.n_bf)) * 0.02
    return A + A.T


@pytest.mark.gpu
@pytest.mark.parametrize("n,basis,spherical", [(1, "cc-pVTZ", True), (1, "cc-pVTZ", False), (2, "cc-pVTZ", False),
                                               (1, "def2-SVP", True), (3, "def2-SVP", False)])
def test_rows_match_the_oracle(cuda_ok, oracle_mod, n, basis, spherical):
    from tonto_b200.fock import TF_JK_J_ONLY, TF_JK_K_ONLY, FockBuilder
    mol = water_cluster(n, seed=31 + n, basis=basis, spherical=spherical)
    Pa, Pb = _density(mol, 1), _density(mol, 2)
    orc = oracle_mod.Oracle(mol, schwarz_cutoff=1e-12)
    fb = FockBuilder(mol, schwarz_cutoff=1e-12)
    want = orc.jk_uhf(Pa, Pb)
    Jr, Kr = orc.jk(Pa)
    for _ in range(2):                               # class by class, then a replayed graph
        for got, ref in zip(fb.make_u_JK(Pa, Pb), want):
            assert np.max(np.abs(got - ref)) <= TOL
    for _ in range(2):
        J, K = fb.make_r_JK(Pa)
        assert np.max(np.abs(J - Jr)) <= TOL and np.max(np.abs(K - Kr)) <= TOL
    J, K = fb.make_r_JK(Pa, TF_JK_J_ONLY)
    assert np.max(np.abs(J - Jr)) <= TOL and not K.any()
    J, K = fb.make_r_JK(Pa, TF_JK_K_ONLY)
    assert np.max(np.abs(K - Kr)) <= TOL and not J.any()
    fb.close()
