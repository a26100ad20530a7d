"""The mesh transforms on every kind of mesh the passes distinguish, against numpy's FFT (needs a B200).

``Engine.pme_potential`` against the same smooth-PME sum (order-4 spread, half-spectrum product,
interpolation) in numpy: odd and even line lengths (rows are transformed in pairs), planes that fit
in shared memory and planes that do not, lengths of one stage and of many, the shortest and the
longest.  Both are FP64 sums of the same terms, so they agree to rounding: the bound is 1e-11 of the
potential's RMS (about 5 log2(N) eps of the transforms, and the condition of the sums).  A context
refilled with another mesh runs the passes for that mesh.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ALPHA = 0.32
K = float(np.float32(1388.431112))  # the engine's Coulomb constant is a float


def bspline(w):
    c = 1.0 - w
    return np.stack([w ** 3 / 6, (-3 * w ** 3 + 3 * w * w + 3 * w + 1) / 6, (3 * w ** 3 - 6 * w * w + 4) / 6,
                     c ** 3 / 6], -1)


def weights(x, start, L, n):
    """Mesh indices [p, 4, 3] and weights [p, 4, 3] of the points."""
    u = (x - start) / L * n
    f = np.floor(u)
    idx = (f.astype(int)[:, None, :] - np.arange(4)[None, :, None]) % n
    return idx, np.moveaxis(bspline(u - f), -1, 1)


def numpy_potential(s, mesh, pts):
    info = s.SimInfo[0]
    L, start, n = info["cryst"].astype(float), info["startxyz"].astype(float), np.array(mesh)
    rows = np.concatenate([np.arange(int(s.fragmentInfo[0]["startRes"]))] + [
        np.arange(int(f["startRes"]), int(f["startRes"]) + int(f["totalNum"])) for f in s.fragmentInfo])
    atoms = np.concatenate([np.arange(r["atomStart"], r["atomStart"] + r["atomNum"]) for r in s.residueInfo[rows]])
    x, q = s.atomInfo["position"][atoms].astype(float), s.atomInfo["charge"][atoms].astype(float)
    Q = np.zeros(mesh)
    idx, w = weights(x, start, L, n)
    for a in range(4):
        for b in range(4):
            for c in range(4):
                np.add.at(Q, (idx[:, a, 0], idx[:, b, 1], idx[:, c, 2]), q * w[:, a, 0] * w[:, b, 1] * w[:, c, 2])
    m = [np.fft.fftfreq(n[0]) * n[0], np.fft.fftfreq(n[1]) * n[1], np.arange(n[2] // 2 + 1)]
    if n[0] % 2 == 0:
        m[0][n[0] // 2] = n[0] // 2
    if n[1] % 2 == 0:
        m[1][n[1] // 2] = n[1] // 2
    mm = sum(np.meshgrid(*[(v / l) ** 2 for v, l in zip(m, L)], indexing="ij"))
    mod = []
    for a in range(3):
        k = np.arange(n[a])
        mod.append(1 / np.abs(sum(c * np.exp(2j * np.pi * k * j / n[a]) for j, c in enumerate((1 / 6, 2 / 3, 1 / 6)))) ** 2)
    with np.errstate(divide="ignore", invalid="ignore"):
        G = K * np.exp(-np.pi ** 2 * mm / float(np.float32(ALPHA)) ** 2) / (np.pi * np.prod(L) * mm)
    G[0, 0, 0] = 0.0
    G *= mod[0][:, None, None] * mod[1][None, :, None] * mod[2][None, None, : n[2] // 2 + 1]
    phi = np.fft.irfftn(np.fft.rfftn(Q) * G, s=mesh, axes=(0, 1, 2)) * np.prod(n)
    idx, w = weights(pts, start, L, n)
    out = np.zeros(len(pts))
    for a in range(4):
        for b in range(4):
            for c in range(4):
                out += phi[idx[:, a, 0], idx[:, b, 1], idx[:, c, 2]] * w[:, a, 0] * w[:, b, 1] * w[:, c, 2]
    return out


def options(mesh, **kw):
    from pygcmc_b200._native import default_options
    o = default_options(pme=1, pme_alpha=ALPHA, **kw)
    for a in range(3):
        o.pme_grid[a] = mesh[a]
    return o


@pytest.mark.parametrize("mesh", [(8, 8, 8), (9, 27, 81), (64, 64, 64), (12, 54, 48), (128, 128, 96), (12, 128, 128),
                                  (8, 243, 162), (256, 9, 12), (16, 256, 256), (27, 16, 243)])
def test_mesh_potential_matches_numpy(water_small, mesh):
    from pygcmc_b200.engine import Engine
    info = water_small.SimInfo[0]
    pts = info["startxyz"].astype(float) + np.random.default_rng(5).random((200, 3)) * info["cryst"].astype(float)
    with Engine(water_small.copy(), options(mesh)) as e:
        phi = e.pme_potential(pts)
    ref = numpy_potential(water_small, mesh, pts)
    assert np.abs(phi - ref).max() <= 1e-11 * np.sqrt((ref ** 2).mean())


def test_refill_with_another_mesh(water_small):
    """The drop-in's kept context, refilled with a larger mesh, gives a fresh context's chain."""
    from pygcmc_b200._native import lib
    from pygcmc_b200.gpu import runGCMC

    def chain(mesh):
        s = water_small.copy()
        s.SimInfo[0]["mcsteps"] = 24
        s.moveArray = s.moveArray[:24].copy()
        runGCMC(*s.arrays(), options=options(mesh))
        return s

    lib().gcmc_release_cache()
    fresh = chain((64, 64, 64))
    lib().gcmc_release_cache()
    for mesh in ((16, 16, 16), (12, 128, 128)):
        chain(mesh)
    again = chain((64, 64, 64))
    assert np.array_equal(fresh.fragmentInfo["totalNum"], again.fragmentInfo["totalNum"])
    assert np.array_equal(fresh.atomInfo["position"], again.atomInfo["position"])
