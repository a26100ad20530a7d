"""The context's scratch when its stream is being captured and when a call fails half-way (needs a B200)."""
import contextlib
import ctypes

import numpy as np
import pytest

from pygcmc_b200 import poses as PZ

pytestmark = pytest.mark.gpu

RELAXED = 2


@contextlib.contextmanager
def _capture(stream):
    """The stream under capture; what was captured, or spoilt by a refused call, is dropped."""
    cu = ctypes.CDLL("libcuda.so.1")
    h, graph = ctypes.c_void_p(stream), ctypes.c_void_p()
    assert cu.cuStreamBeginCapture_v2(h, RELAXED) == 0
    yield
    cu.cuStreamEndCapture(h, ctypes.byref(graph))
    if graph:
        cu.cuGraphDestroy(graph)


def _poses(s, n):
    tpl, q, t = PZ.template(s, 2)
    com, quat = PZ.random_poses(s, n, seed=n)
    return PZ.rigid_sites(tpl, com, quat).astype(np.float32), q, t, com.astype(np.float32)


def test_explicit_poses_on_a_captured_stream(protein_small):
    """A call that waits for its results cannot be captured: refused, with a small scratch and with one that
    would have to grow, and the calls after the capture give what they gave before."""
    import torch
    from pygcmc_b200._native import GcmcError
    from pygcmc_b200.engine import Engine
    stream = torch.cuda.Stream()
    with Engine(protein_small.copy(), stream=stream.cuda_stream) as e:
        with Engine(protein_small.copy()) as other:
            want = {n: other.energy_poses(*_poses(protein_small, n)) for n in (4, 3000, 9000)}
        for n in (4, 3000, 9000):
            with _capture(stream.cuda_stream):
                with pytest.raises(GcmcError):
                    e.energy_poses(*_poses(protein_small, n))
            for m in (n, 3000):
                got = e.energy_poses(*_poses(protein_small, m))
                assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(got, want[m]))


def test_gradients_on_a_stream_that_joins_a_capture(protein_small):
    """Gradients on another stream than the context's, whose own stream is being captured: the call joins the
    capture, with memory of its own, and nothing of the graph is left in the context."""
    import torch
    from pygcmc_b200._native import lib
    from pygcmc_b200.engine import Engine
    stream, side = torch.cuda.Stream(), torch.cuda.Stream()
    xyz, q, t, cen = _poses(protein_small, 3000)
    d = [torch.tensor(a, device="cuda") for a in (xyz, q, t, cen)]
    out = torch.zeros((2, 3000), dtype=torch.float64, device="cuda")
    gx = torch.empty(xyz.shape, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()

    def call(e, row):
        p = [ctypes.c_void_p(a.data_ptr()) for a in d]
        return lib().gcmc_energy_grad(e.handle, 0, p[0], p[1], p[2], t.ctypes.data_as(ctypes.c_void_p), xyz.shape[1],
                                      p[3], None, len(xyz), None, None, ctypes.c_void_p(out[row].data_ptr()),
                                      ctypes.c_void_p(gx.data_ptr()), None, None, ctypes.c_void_p(side.cuda_stream))
    with Engine(protein_small.copy(), stream=stream.cuda_stream) as e:
        with _capture(stream.cuda_stream):
            assert call(e, 0) == 0
        assert call(e, 1) == 0
        torch.cuda.synchronize()
        want, _ = e.energy_poses(xyz, q, t, cen)
        assert np.array_equal(out[1].cpu().numpy(), want, equal_nan=True)
        assert not out[0].any()  # captured, and never launched


def test_failed_gradients_keep_their_place(protein_small):
    """A gradient call that fails after its first launches (here on the error of a call before it) still has the
    context's stream wait for them, as they use the scratch that the next call takes."""
    import torch
    from pygcmc_b200._native import lib
    from pygcmc_b200.engine import Engine
    stream, side = torch.cuda.Stream(), torch.cuda.Stream()
    xyz, q, t, cen = _poses(protein_small, 64)
    d = [torch.tensor(a, device="cuda") for a in (xyz, q, t, cen)]
    out = torch.empty(64, dtype=torch.float64, device="cuda")
    done = torch.cuda.Event()
    with Engine(protein_small.copy(), stream=stream.cuda_stream) as e:
        want, _ = e.energy_poses(xyz, q, t, cen)
        torch.cuda.synchronize()
        with _capture(stream.cuda_stream):
            assert lib().gcmc_sync(e.handle) == 1
        p = [ctypes.c_void_p(a.data_ptr()) for a in d]
        with torch.cuda.stream(side):
            torch.cuda._sleep(1_000_000_000)  # about half a second
            st = lib().gcmc_energy_grad(e.handle, 0, p[0], p[1], p[2], t.ctypes.data_as(ctypes.c_void_p), xyz.shape[1],
                                        p[3], None, 64, None, None, ctypes.c_void_p(out.data_ptr()), None, None, None,
                                        ctypes.c_void_p(side.cuda_stream))
            done.record()
        assert st == 1
        assert not done.query()
        got, _ = e.energy_poses(xyz, q, t, cen)
        assert done.query()
        assert np.array_equal(got, want, equal_nan=True)
        torch.cuda.synchronize()


def test_scratch_is_given_back(protein_small):
    """gcmc_release_cache frees the large scratch of a context in use, and the context works on; with other
    contexts made and closed before it."""
    import torch
    from pygcmc_b200._native import lib
    from pygcmc_b200.engine import Engine
    n = 120000
    xyz, q, t, cen = (torch.tensor(a, device="cuda") if i != 2 else a for i, a in enumerate(_poses(protein_small, n)))
    tt = torch.tensor(t, device="cuda")
    out = torch.empty((3,) + xyz.shape, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()

    def call(e, row):
        p = [ctypes.c_void_p(a.data_ptr()) for a in (xyz, q, tt, cen)]
        assert lib().gcmc_energy_grad(e.handle, 0, p[0], p[1], p[2], t.ctypes.data_as(ctypes.c_void_p), xyz.shape[1],
                                      p[3], None, n, None, None, None, ctypes.c_void_p(out[row].data_ptr()), None,
                                      None, None) == 0
        e.sync()

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]
    Engine(protein_small.copy()).close()
    with Engine(protein_small.copy()) as e:
        call(e, 0)  # (the kernel's one-time device memory)
        held = 32 * n * xyz.shape[1]
        assert 8 << 20 < held < 64 << 20
        before = free()
        assert lib().gcmc_release_cache() == 0
        e.sync()
        assert free() - before > held // 2
        call(e, 1)
        assert lib().gcmc_release_cache() == 0  # while its launches may run
        call(e, 2)
    assert lib().gcmc_release_cache() == 0
    a, b, c = (v.cpu().numpy() for v in out)
    assert np.array_equal(a, b, equal_nan=True) and np.array_equal(a, c, equal_nan=True)
