"""The drop-in runs a chain in chunks that speculate or not (needs a B200).

Whatever the chunks' modes and however the run's length falls on them, runGCMC's final state is the
sequential engine's bit for bit, on a system whose steps mostly accept (water) and one that
speculates after its first chunks (the protein continued, few steps accepting).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same(a, b):
    assert np.array_equal(a.fragmentInfo["totalNum"], b.fragmentInfo["totalNum"])
    for f in a.fragmentInfo:
        r = a.residueInfo[int(f["startRes"]):int(f["startRes"]) + int(f["totalNum"])]
        if len(r):
            s = slice(int(r["atomStart"].min()), int((r["atomStart"] + r["atomNum"]).max()))
            assert np.array_equal(a.atomInfo["position"][s], b.atomInfo["position"][s])


@pytest.mark.parametrize("which", ["protein_small", "water_small"])
@pytest.mark.parametrize("n", [1, 7, 24, 25, 32, 33, 64, 97, 200])
@pytest.mark.parametrize("kernel", [0, 1], ids=["per_pose", "tiled"])
def test_dropin_equals_sequential_engine(request, which, n, kernel):
    from pygcmc_b200._native import default_options
    from pygcmc_b200.engine import Engine
    from pygcmc_b200.gpu import runGCMC
    s = request.getfixturevalue(which).copy()
    s.SimInfo[0]["mcsteps"] = n
    s.moveArray = s.moveArray[:n].copy()
    with Engine(s.copy(), default_options(speculate=-1, energy_kernel=kernel)) as e:
        e.run(n)
        e.sync()
        want = e.download()
    got = s.copy()
    runGCMC(*got.arrays(), options=default_options(energy_kernel=kernel))
    same(want, got)


def test_long_run_switches_modes():
    """600 steps of a protein whose insertions are mostly rejected (chemical potentials -8 lower)."""
    from pygcmc_b200 import system as S
    from pygcmc_b200._native import default_options
    from pygcmc_b200.engine import Engine
    from pygcmc_b200.gpu import runGCMC
    s = S.protein_system(seed=5, n_atoms=3000, box=48.0, radius=18.0, mcsteps=600, conf_bias=256, muex_shift=-8.0)
    with Engine(s.copy(), default_options(speculate=-1, log_steps=600, log_kmax=1)) as e:
        e.run(600)
        e.sync()
        want = e.download()
        accepted = e.logs()[0]["n_accept"] > 0
    # several chunks have at least 11 in 20 steps without an acceptance, so both loops run
    quiet = [(~accepted[i:i + 32]).mean() for i in range(0, 576, 32)]
    assert max(quiet[:-2]) >= 0.55
    got = s.copy()
    runGCMC(*got.arrays())
    same(want, got)
