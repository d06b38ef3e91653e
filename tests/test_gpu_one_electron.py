"""One-electron integrals and Schwarz bounds (a warp a shell pair) against the oracle: pairs
with fewer and more primitive pairs than lanes, every pair class up to f, Cartesian and
spherical, single and batched contexts, and symmetric to the bit."""

import numpy as np
import pytest

from tonto_b200.molecules import alkane, water_cluster


@pytest.mark.gpu
@pytest.mark.parametrize("basis,spherical", [("STO-3G", True), ("6-31G(d)", False), ("cc-pVDZ", True),
                                             ("cc-pVTZ", False)])
def test_one_electron_and_schwarz(cuda_ok, oracle_mod, basis, spherical):
    from tonto_b200.fock import BatchFockBuilder, FockBuilder
    mols = [water_cluster(n, seed=50 + n, basis=basis, spherical=spherical) for n in (1, 3)]
    if basis == "6-31G(d)":
        mols.append(alkane(3, seed=1, basis=basis, spherical=spherical))
    batch = BatchFockBuilder(mols)
    Sb, Tb, Vb = batch.one_electron()
    batch.close()
    for i, mol in enumerate(mols):
        orc = oracle_mod.Oracle(mol)
        fb = FockBuilder(mol)
        mr = orc.max_I()
        assert np.max(np.abs(fb.max_I - mr) / np.maximum(mr, 1e-300)) <= 1e-12
        for got, in_batch, ref in zip(fb.one_electron(), (Sb[i], Tb[i], Vb[i]), orc.one_electron()):
            # elements up to some 1e2; the bar of the f-shell tests
            assert np.max(np.abs(got - ref)) < 1e-11 and np.max(np.abs(in_batch - ref)) < 1e-11
            if not spherical:
                assert np.array_equal(got, got.T)
        fb.close()
