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


def test_no_graph_of_another_shape(protein_small):
    """A kept batch context whose calls go from a graph of one kernel to the persistent loop of another and from
    there to a graph of that kernel: each call gives the chains of a fresh context."""
    from pygcmc_b200._native import default_options, lib
    from pygcmc_b200.engine import Engine
    from pygcmc_b200.gpu import runGCMC_batch
    n = 48

    def replicas():
        out = []
        for r in range(2):
            s = protein_small.copy()
            s.SimInfo = s.SimInfo.copy()
            s.SimInfo[0]["mcsteps"] = n
            s.SimInfo[0]["seed"] = 17 + r
            s.moveArray = np.ascontiguousarray(s.moveArray[:n])
            out.append(s)
        return out
    assert lib().gcmc_release_cache() == 0
    for kernel, persistent in ((1, 0), (0, 1), (0, 0), (1, 0), (0, 1), (1, 0)):
        opts = default_options(energy_kernel=kernel, persistent=persistent)
        got = replicas()
        runGCMC_batch(got, opts)
        with Engine(replicas(), opts) as e:
            e.run(n)
            e.sync()
            for r, s in enumerate(got):
                want = e.download(r)
                assert np.array_equal(s.fragmentInfo["totalNum"], want.fragmentInfo["totalNum"])
                for f in want.fragmentInfo:
                    a, b = int(f["startRes"]), int(f["startRes"]) + int(f["totalNum"])
                    assert np.array_equal(s.residueInfo["position"][a:b], want.residueInfo["position"][a:b])
    assert lib().gcmc_release_cache() == 0
