"""Inputs that a context's set-up refuses, and what the same thread does next (needs a B200)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ARG, LIMIT = 2, 3


def _good(s):
    from pygcmc_b200._native import default_options
    from pygcmc_b200.engine import Engine
    with Engine(s.copy(), default_options()) as e:
        e.run(40)
        e.sync()
        return e.download()


def _mesh(n):
    from pygcmc_b200._native import default_options
    o = default_options(pme=1)
    for a in range(3):
        o.pme_grid[a] = n
    return o


@pytest.mark.parametrize("how", ["mesh_factor", "mesh_small", "bits_header"])
def test_refused_context_leaves_nothing_behind(protein_small, how):
    """A mesh edge that is not 2^a 3^b, one below 8, a grid record with a voxel edge of zero: refused with the
    status of the header, by a new context as by the first call of the drop-in and of the batch; the next context
    of the thread is created and runs the same chain as one before."""
    from pygcmc_b200 import _native as N
    from pygcmc_b200.engine import Engine
    from pygcmc_b200.gpu import runGCMC, runGCMC_batch
    s = protein_small
    before = _good(s)
    assert N.lib().gcmc_release_cache() == 0  # the calls below make contexts of their own
    bad = s.copy()
    grid = bad.grid
    if how == "bits_header":
        opts, status = N.default_options(grid_bits=1), ARG
        grid = bad.grid_bits.copy()
        grid[24:32] = np.frombuffer(np.float64(0.0).tobytes(), np.uint8)  # dx
    else:
        opts, status = (_mesh(50), LIMIT) if how == "mesh_factor" else (_mesh(6), ARG)
    arrays = (bad.SimInfo, bad.fragmentInfo, bad.residueInfo, bad.atomInfo, grid, bad.ff, bad.moveArray)
    calls = [lambda: runGCMC(*arrays, options=opts), lambda: runGCMC_batch([arrays, arrays], opts)]
    if how != "bits_header":
        calls.append(lambda: Engine(bad, opts))
    for call in calls:
        for _ in range(2):
            with pytest.raises(N.GcmcError) as err:
                call()
            assert err.value.status == status
        after = _good(s)
        assert np.array_equal(before.fragmentInfo["totalNum"], after.fragmentInfo["totalNum"])
        assert np.array_equal(before.atomInfo["position"], after.atomInfo["position"])
