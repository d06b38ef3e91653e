"""A replayed build launches the kernels for the lists it has: a graph captured after short
lists (a nearly empty density, a density change) is right on long ones, which then run the
lane groups that share quartets, and the builds after it run the kernels for long lists."""

import re

import numpy as np
import pytest

from tonto_b200.molecules import water_cluster

TOL = 1e-11          # the element bar of every FP64 build


def _kernels(build):
    """Names of the (pp|pp) kernels that build() launches."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        build()
        torch.cuda.synchronize()
    names = [e.name() for e in prof.profiler.kineto_results.events()]
    if not any("k_jk" in n for n in names):
        pytest.skip("the profiler does not see kernels here")
    return {m.group(0) for n in names for m in [re.search(r"k_jk(?:_rows)?<1, 1, 1, 1,[^>]*>", n)] if m}


@pytest.mark.gpu
@pytest.mark.parametrize("first", ["nearly empty", "change"])
def test_long_lists_after_short_ones(cuda_ok, oracle_mod, first):
    from tonto_b200.fock import TF_JK_DELTA, TF_JK_MIXED, FockBuilder
    mol = water_cluster(6, seed=9)                   # some 40000 (pp|pp) quartets, the line is at 8192
    n = mol.n_bf
    A = np.random.default_rng(13).normal(size=(n, n)) * 0.03
    P = A + A.T
    Jr, Kr = oracle_mod.Oracle(mol, schwarz_cutoff=1e-12).jk(P)
    fb = FockBuilder(mol, schwarz_cutoff=1e-12)
    flags = TF_JK_MIXED | TF_JK_DELTA
    scale = 1e-9 if first == "nearly empty" else 1e-3
    fb.make_r_JK(P)                                  # sizes the list
    assert all(k.startswith("k_jk<") for k in _kernels(lambda: fb.make_r_JK(P)))
    for _ in range(2):
        if first == "nearly empty":
            fb.set_graph(True)                       # (the next build captures)
            fb.make_r_JK(scale * P)
        else:
            fb.make_r_JK(scale * P, flags)
    for _ in range(3):
        J, K = fb.make_r_JK(P)
        assert fb.stats()["graph"] == 1
        assert np.max(np.abs(J - Jr)) <= TOL and np.max(np.abs(K - Kr)) <= TOL
    last = _kernels(lambda: fb.make_r_JK(P))
    assert last and all(k.startswith("k_jk<") for k in last), last
    fb.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n,basis", [(6, "cc-pVDZ"), (2, "cc-pVTZ")])
def test_graph_captured_on_a_nearly_empty_build(cuda_ok, oracle_mod, n, basis):
    # no build of full length before the capture: its first replay on the full lists runs every
    # class as captured for almost none, the next one is captured anew
    from tonto_b200.fock import FockBuilder
    mol = water_cluster(n, seed=9, basis=basis)
    A = np.random.default_rng(17).normal(size=(mol.n_bf, mol.n_bf)) * 0.03
    P = A + A.T
    Jr, Kr = oracle_mod.Oracle(mol, schwarz_cutoff=1e-12).jk(P)
    fb = FockBuilder(mol, schwarz_cutoff=1e-12)
    fb.make_r_JK(P)                                  # sizes the list
    fb.set_shard(0, 1)                               # and forgets its lengths
    seen = []
    for k in range(4):
        seen.append(_kernels(lambda: fb.make_r_JK(1e-9 * P if k == 0 else P)))
        if k > 0:
            J, K = fb.make_r_JK(P)
            assert fb.stats()["graph"] == 1
            assert np.max(np.abs(J - Jr)) <= TOL and np.max(np.abs(K - Kr)) <= TOL
    if basis == "cc-pVDZ":
        assert any(k.startswith("k_jk_rows<1, 1, 1, 1, 4, true") for k in seen[1])   # sharing, on the long list
        assert seen[3] and all(k.startswith("k_jk<") for k in seen[3])
    fb.close()
