"""The autotuner changes a context only when it has succeeded: after a refused density, and
where no schedule can be timed, the context launches what it launched before."""

import math
import re

import numpy as np
import pytest

from tonto_b200.molecules import water_cluster


def _launches(build):
    """(kernel, stream) of every quartet kernel that build() launches."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        build()
        torch.cuda.synchronize()
    out = []
    for e in prof.profiler.kineto_results.events():
        m = re.search(r"k_jk(?:_rows)?<[^>]*>", e.name())
        if m:
            out.append((m.group(0), e.device_resource_id()))
    if not out:
        pytest.skip("the profiler does not see kernels here")
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("why", ["refused", "chunked"])
def test_context_is_as_it_was(cuda_ok, why):
    import torch
    from tonto_b200.fock import FockBuilder, TontoFockError
    mol = water_cluster(4, seed=7)
    n = mol.n_bf
    A = np.random.default_rng(11).normal(size=(n, n)) * 0.05
    P = torch.tensor(A + A.T, device="cuda:0")
    J, K = torch.empty_like(P), torch.empty_like(P)
    fb = FockBuilder(mol, schwarz_cutoff=1e-12)
    fb.make_r_JK_device(P, J, K)                     # (the first build loads the kernels)
    fb.close()
    fb = FockBuilder(mol, schwarz_cutoff=1e-12)
    fb.set_list_budget(1 << 10)                      # lists too long for one chunk: class launches, no graph
    before = _launches(lambda: fb.make_r_JK_device(P, J, K))
    if why == "refused":
        bad = P.clone()
        bad[2, 3] = bad[3, 2] = math.nan
        with pytest.raises(TontoFockError):
            fb.autotune(bad, J, K)
        fb.make_r_JK_device(P, J, K)
        after = _launches(lambda: fb.make_r_JK_device(P, J, K))
        assert sorted(k for k, _ in after) == sorted(k for k, _ in before)
    else:
        tune = fb.autotune(P, J, K)
        assert tune["candidates"] == 0
        after = _launches(lambda: fb.make_r_JK_device(P, J, K))
    assert len({s for _, s in before}) > 1 and len({s for _, s in after}) > 1
    Jr, Kr = J.clone(), K.clone()
    fb.close()
    fb = FockBuilder(mol, schwarz_cutoff=1e-12)
    fb.make_r_JK_device(P, J, K)
    assert (J - Jr).abs().max() < 1e-11 and (K - Kr).abs().max() < 1e-11
    fb.close()
