"""Explicit-pose calls of every size class (needs a B200).

gcmc_energy_poses sends its poses in blocks of 2048 through kept scratch and picks the number of
work items per pose from their count; the gradient entry point shares that scratch.  Whatever the
count, each pose's energy is the same sum of the same FP32 atom terms in FP64, in another order: the
results agree with one-pose calls within 64 eps of the pose's sum of |terms|, and the group counts
are equal.  A call that grows the scratch, and calls of another context between, change nothing.
"""
import numpy as np
import pytest

from pygcmc_b200 import poses as PZ

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 37, 2047, 2048, 2049, 6001])
@pytest.mark.parametrize("skip", [False, True])
def test_energy_poses_blocks(oracle_lib, protein_small, n, skip):
    from pygcmc_b200.engine import Engine
    s = protein_small
    tpl, q, t = PZ.template(s, 2)
    com, quat = PZ.random_poses(s, n, seed=n)
    xyz = PZ.rigid_sites(tpl, com, quat).astype(np.float32)
    cen = com.astype(np.float32)
    self_res = None
    if skip:
        self_res = np.random.default_rng(n).integers(-1, int(s.fragmentInfo[0]["startRes"]), n).astype(np.int32)
    pick = np.unique(np.linspace(0, n - 1, min(n, 24)).astype(int))
    with Engine(s.copy()) as e:
        small, ng_small = e.energy_poses(xyz[:1], q, t, cen[:1], None if self_res is None else self_res[:1])
        big, ng_big = e.energy_poses(xyz, q, t, cen, self_res)
        again, _ = e.energy_poses(xyz, q, t, cen, self_res)
        one = [e.energy_poses(xyz[i:i + 1], q, t, cen[i:i + 1], None if self_res is None else self_res[i:i + 1])
               for i in pick]
    assert np.array_equal(big, again, equal_nan=True)
    l1 = oracle_lib.energy_batch(s, xyz[pick], q, t, cen[pick], None if self_res is None else self_res[pick], mode=0,
                                 want_l1=True)[3]
    e1 = np.array([x[0][0] for x in one])
    assert np.array_equal(np.isfinite(big[pick]), np.isfinite(e1))
    ok = np.isfinite(e1)
    assert np.all(np.abs(big[pick][ok] - e1[ok]) <= 64 * np.finfo(float).eps * l1[ok])
    assert np.array_equal(ng_big[pick], [x[1][0] for x in one]) and ng_small[0] == ng_big[0]


def test_scratch_shared_by_streams_and_calls(protein_small):
    """Gradient calls on two streams and host calls between them share the context's scratch."""
    import torch
    from pygcmc_b200.engine import Engine
    from pygcmc_b200.grad import pose_energy
    s = protein_small
    tpl, q, t = PZ.template(s, 2)
    dev = torch.device("cuda")

    def inputs(n):
        com, quat = PZ.random_poses(s, n, seed=n)
        return PZ.rigid_sites(tpl, com, quat).astype(np.float32), com.astype(np.float32)

    def grads(eng, x, c, stream):
        with torch.cuda.stream(stream):
            X = torch.tensor(x, device=dev, requires_grad=True)
            F = torch.tensor(s.ff, device=dev)
            E = pose_energy(eng, 0, X, torch.tensor(q, device=dev), F, t, centres=torch.tensor(c, device=dev))
            torch.nan_to_num(E, posinf=0.0, neginf=0.0).sum().backward()
            return E, X.grad

    sizes = [5, 700, 64, 3000, 2, 1500]
    with Engine(s.copy()) as e:
        alone = []
        for n in sizes:
            r = grads(e, *inputs(n), torch.cuda.current_stream())
            torch.cuda.synchronize()
            alone.append([v.detach().cpu().numpy() for v in r])
    with Engine(s.copy()) as e:
        streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        got = []
        for i, n in enumerate(sizes):
            x, c = inputs(n)
            got.append(grads(e, x, c, streams[i % 2]))
            if i % 2:
                e.energy_poses(x, q, t, c)
        torch.cuda.synchronize()
        for a, b in zip(alone, got):
            for u, v in zip(a, b):
                assert np.array_equal(u, v.detach().cpu().numpy(), equal_nan=True)
