"""What a run enqueues, whatever step it starts at (needs a B200)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [0, 1], ids=["per_pose", "tiled"])
def test_runs_capture_nothing(protein_small, kernel):
    """The step loop's graphs are made with the context: a run from an odd or an even step, a long or a short one,
    launches them and makes none, and the chain is the one of a single run."""
    import torch
    from pygcmc_b200._native import default_options
    from pygcmc_b200.engine import Engine
    opts = default_options(energy_kernel=kernel)
    runs = [1, 2, 33, 1, 5, 40, 18]
    with Engine(protein_small.copy(), opts) as e:
        e.run(sum(runs))
        e.sync()
        whole = e.download()
    with Engine(protein_small.copy(), opts) as e:
        e.sync()
        names = []
        for n in runs:
            with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA,
                                                    torch.profiler.ProfilerActivity.CPU]) as prof:
                e.run(n)
                e.sync()
            names.append({ev.name for ev in prof.events()})
        parts = e.download()
    for n, seen in zip(runs, names):
        assert "cudaGraphLaunch" in seen, (n, sorted(seen))
        made = [x for x in seen if "Instantiate" in x or "Capture" in x]
        assert not made, (n, made)
    assert np.array_equal(whole.fragmentInfo["totalNum"], parts.fragmentInfo["totalNum"])
    assert np.array_equal(whole.atomInfo["position"], parts.atomInfo["position"])
    assert np.array_equal(whole.residueInfo["position"], parts.residueInfo["position"])
