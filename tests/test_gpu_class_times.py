"""Per-class device times of direct builds: a context's first build and builds whose list is
chunked launch class by class, on branches that overlap, and report each class's time."""

import numpy as np
import pytest

from tonto_b200.molecules import water_cluster


@pytest.mark.gpu
@pytest.mark.parametrize("budget", [None, 1 << 12, 1])       # one chunk, several, one class pair each
@pytest.mark.parametrize("graph", [True, False])
def test_direct_builds_report_class_times(cuda_ok, budget, graph):
    from tonto_b200.fock import FockBuilder
    mol = water_cluster(3, seed=2)
    A = np.random.default_rng(3).normal(size=(mol.n_bf, mol.n_bf)) * 0.05
    fb = FockBuilder(mol, schwarz_cutoff=1e-12)
    fb.set_graph(graph)
    if budget:
        fb.set_list_budget(budget)
    for _ in range(2):
        fb.make_r_JK(A + A.T)
        st, cls = fb.stats(), fb.class_stats()
        if st["graph"]:
            assert budget is None and graph and all(c["ms"] == 0.0 for c in cls) and st["eri_ms"] == st["build_ms"]
            continue
        assert len(cls) > 10 and all(c["ms"] > 0.0 for c in cls)
        total = sum(c["ms"] for c in cls)
        # (event times have a resolution of half a microsecond)
        slack = 1e-3 * len(cls)
        assert max(c["ms"] for c in cls) <= st["eri_ms"] + slack and st["eri_ms"] <= st["build_ms"] + slack
        if not graph:
            assert abs(st["eri_ms"] - total) <= slack
    fb.close()
