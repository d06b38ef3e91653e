"""Classes with two kinds of kernels, a thread a quartet for long lists and lane groups for
short ones: both kinds, plain and deterministic, restricted and unrestricted."""

import numpy as np
import pytest

from tonto_b200.molecules import water_cluster

TOL = 1e-11          # the element bar of every FP64 build; densities of order 0.1


def _density(mol, seed):
    A = np.random.default_rng(seed).normal(size=(mol.n_bf, mol.n_bf)) * 0.02
    return A + A.T


@pytest.mark.gpu
@pytest.mark.parametrize("n,basis,spherical", [(1, "STO-3G", True), (2, "STO-3G", True), (1, "cc-pVTZ", True),
                                               (1, "cc-pVTZ", False), (2, "def2-SVP", False)])
def test_thread_kernels_on_short_lists(cuda_ok, oracle_mod, n, basis, spherical):
    # a deterministic build takes the thread kernels whatever the lists hold
    from tonto_b200.fock import FockBuilder
    mol = water_cluster(n, seed=41 + n, basis=basis, spherical=spherical)
    Pa, Pb = _density(mol, 3), _density(mol, 4)
    orc = oracle_mod.Oracle(mol, schwarz_cutoff=1e-12)
    fb = FockBuilder(mol, schwarz_cutoff=1e-12, deterministic=True)
    for got, ref in zip(fb.make_r_JK(Pa), orc.jk(Pa)):
        assert np.max(np.abs(got - ref)) <= TOL
    for _ in range(2):
        for got, ref in zip(fb.make_u_JK(Pa, Pb), orc.jk_uhf(Pa, Pb)):
            assert np.max(np.abs(got - ref)) <= TOL
    fb.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n,basis", [(2, "cc-pVTZ"), (4, "cc-pVTZ"), (6, "def2-SVP")])
def test_plain_and_deterministic_agree(cuda_ok, n, basis):
    # lists from a few hundred to 80000 quartets: on both sides of the line
    from tonto_b200.fock import FockBuilder
    mol = water_cluster(n, seed=51 + n, basis=basis)
    Pa, Pb = _density(mol, 5), _density(mol, 6)
    out = []
    for det in (False, True):
        fb = FockBuilder(mol, schwarz_cutoff=1e-12, deterministic=det)
        for _ in range(2):
            got = [*fb.make_r_JK(Pa), *fb.make_u_JK(Pa, Pb)]
        out.append(got)
        fb.close()
    for x, y in zip(*out):
        assert np.max(np.abs(x - y)) <= TOL
