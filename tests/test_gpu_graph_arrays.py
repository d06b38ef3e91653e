"""Replayed builds of changing arrays: a captured build serves any density, J and K arrays, and
restricted and unrestricted builds of one context keep a graph each."""

import numpy as np
import pytest

from tonto_b200.molecules import water_cluster

TOL = 1e-11          # the element bar of every FP64 build; densities of order 0.1


def _captures(builds):
    """Graphs instantiated while builds() runs."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        builds()
        torch.cuda.synchronize()
    names = [e.name() for e in prof.profiler.kineto_results.events()]
    if not any("cudaGraphLaunch" in n for n in names):
        pytest.skip("the profiler does not see the runtime's calls here")
    return sum("GraphInstantiate" in n for n in names)


@pytest.mark.gpu
@pytest.mark.parametrize("basis,spherical", [("STO-3G", True), ("cc-pVDZ", True), ("6-31G(d)", False)])
@pytest.mark.parametrize("deterministic", [False, True])
def test_one_graph_serves_any_arrays(cuda_ok, oracle_mod, basis, spherical, deterministic):
    import torch
    from tonto_b200.fock import FockBuilder
    mol = water_cluster(2, seed=3, basis=basis, spherical=spherical)
    n = mol.n_bf
    rng = np.random.default_rng(5)
    dens = []
    for _ in range(4):
        A = rng.normal(size=(n, n)) * 0.05
        dens.append(A + A.T)
    orc = oracle_mod.Oracle(mol, schwarz_cutoff=1e-12)
    fb = FockBuilder(mol, schwarz_cutoff=1e-12, deterministic=deterministic)
    dev = torch.device("cuda", 0)
    sets = []                                                 # arrays of their own for every density
    for i, P in enumerate(dens):
        out = [torch.full((n, n), float("nan"), dtype=torch.float64, device=dev) for _ in range(4)]
        sets.append((torch.tensor(P, device=dev), torch.tensor(dens[i - 1], device=dev), out))
    want = [(orc.jk(P), orc.jk_uhf(P, dens[i - 1])) for i, P in enumerate(dens)]

    def builds(check):
        for (Pa, Pb, out), (ref_r, ref_u) in zip(sets, want):
            for got in out:
                got.fill_(float("nan"))
            fb.make_r_JK_device(Pa, out[0], out[1])
            if check:
                for got, ref in zip(out[:2], ref_r):
                    assert np.max(np.abs(got.cpu().numpy().T - ref)) <= TOL
            fb.make_u_JK_device(Pa, Pb, *out)
            if check:
                assert fb.stats()["graph"] == 1
                for got, ref in zip(out, ref_u):
                    assert np.max(np.abs(got.cpu().numpy().T - ref)) <= TOL
        fb.make_r_JK(dens[0])                                 # the host entry point's own arrays
        fb.make_u_JK(dens[0], dens[1])

    builds(False)                                             # sizes the list, captures both graphs
    builds(True)
    assert _captures(lambda: builds(False)) == 0
    fb.close()
