"""Differentiable pose energies (PyTorch autograd over gcmc_energy_grad).

:class:`PoseEnergy` maps explicit poses -- site coordinates, site charges and
the LJ pair table in the reference's layout (sigma [nm], eps [kJ/mol] per
(site type, atom type); gcmc/cpp/gcmc_energy.h:160-161) -- to the FP64 pose
energies of the engine's kernels, and its backward calls the hand-written
gradient kernel.  :class:`RigidFragment` builds the sites of a fragment type
from a centre of mass and a quaternion, and :func:`lj_table` the pair table
from per-type CHARMM parameters with the reference's combining rule
(gcmc/python/simulation.py:56-75), so that autograd reaches
d E / d(centre of mass, quaternion, eps, rmin/2, site charges).

The environment (fixed atoms and occupied fragment slots of the replica) is
the engine's current state and carries no gradient.  Group inclusion is by
pose centre (the centre of mass), a hard cutoff: E is smooth in the site
coordinates and parameters, piecewise constant in which groups count.
"""
import ctypes

import numpy as np
import torch

from . import values as V
from ._native import check, lib


def _dense(t):
    """t with its elements in order in memory and no negation left to a view's bit: what a raw
    pointer stands for."""
    return t.resolve_neg().contiguous()


def _p(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def _stream():
    """torch's current stream as a cudaStream_t.  torch reports the legacy
    default stream as 0, which the C ABI reads as "the context's stream"; pass
    cudaStreamLegacy (0x1) instead so the kernels stay ordered with torch's work."""
    h = torch.cuda.current_stream().cuda_stream
    return ctypes.c_void_p(h if h else 1)


# Up to this many poses the gradients' chain rule is one kernel (k_pose_chain), whose sum over the
# poses is one block per site.  8 sites, us by the kernel and by the six tensor operations: 64 poses
# 26 and 60, 16384 22 and 61, 65536 33 and 45; beyond, the operations' split reduction is the faster.
CHAIN_POSES = 65536


class PoseEnergy(torch.autograd.Function):
    """E[p] (float64) of poses ``xyz`` [P, ns, 3] float32 with charges ``q`` [ns]
    float32 and pair table ``ff`` [ffX*ffY*2] float32 (all CUDA); ``centres``
    [P, 3] float32 selects the included groups (no gradient)."""

    @staticmethod
    def forward(ctx, xyz, q, ff, centres, engine, rep, site_type, site_type_dev, self_res):
        xyz, q, ff, centres = (_dense(t) for t in (xyz, q, ff, centres))
        P, ns = xyz.shape[0], xyz.shape[1]
        E = torch.empty(P, dtype=torch.float64, device=xyz.device)
        check(lib().gcmc_energy_grad(engine.handle, rep, _p(xyz), _p(q), _p(site_type_dev),
                                     site_type.ctypes.data_as(ctypes.c_void_p), ns, _p(centres), _p(self_res), P,
                                     _p(ff), None, _p(E), None, None, None, _stream()), "gcmc_energy_grad")
        ctx.save_for_backward(xyz, q, ff, centres)
        ctx.engine, ctx.rep, ctx.site_type, ctx.site_type_dev, ctx.self_res = (engine, rep, site_type,
                                                                                site_type_dev, self_res)
        return E

    @staticmethod
    def backward(ctx, gE):
        xyz, q, ff, centres = ctx.saved_tensors
        P, ns = xyz.shape[0], xyz.shape[1]
        gE = _dense(gE.detach().to(torch.float64))
        need_x, need_q, need_ff = ctx.needs_input_grad[0], ctx.needs_input_grad[1], ctx.needs_input_grad[2]
        gxyz = torch.empty((P, ns, 3), dtype=torch.float64, device=xyz.device) if need_x else None
        gq = torch.empty((P, ns), dtype=torch.float64, device=xyz.device) if need_q else None
        gff = torch.zeros(ff.shape[0], dtype=torch.float64, device=xyz.device) if need_ff else None
        if need_x or need_q or need_ff:
            check(lib().gcmc_energy_grad(ctx.engine.handle, ctx.rep, _p(xyz), _p(q), _p(ctx.site_type_dev),
                                         ctx.site_type.ctypes.data_as(ctypes.c_void_p), ns, _p(centres),
                                         _p(ctx.self_res), P, _p(ff), _p(gE), None, _p(gxyz), _p(gq), _p(gff),
                                         _stream()), "gcmc_energy_grad")
        if P <= CHAIN_POSES:
            gx, gqs, gf = (torch.empty(shape, dtype=torch.float32, device=xyz.device) if need else None
                           for need, shape in ((need_x, (P, ns, 3)), (need_q, (ns,)), (need_ff, ff.shape)))
            check(lib().gcmc_pose_chain(_p(gE), _p(gxyz), _p(gq), _p(gff), P, ns, ff.shape[0], _p(gx), _p(gqs),
                                        _p(gf), _stream()), "gcmc_pose_chain")
            return gx, gqs, gf, None, None, None, None, None, None
        gx = (gxyz * gE[:, None, None]).to(xyz.dtype) if need_x else None
        gqs = (gq * gE[:, None]).sum(0).to(q.dtype) if need_q else None
        gf = gff.to(ff.dtype) if need_ff else None
        return gx, gqs, gf, None, None, None, None, None, None


def pose_energy(engine, rep, xyz, q, ff, site_type, centres=None, self_res=None):
    """Differentiable E[p] for sites ``xyz`` [P, ns, 3] (any float dtype; the
    kernels see float32), charges ``q`` [ns], table ``ff``; ``site_type`` a
    numpy int32 array [ns].  ``centres`` defaults to the site centroids."""
    dev = xyz.device
    st = np.ascontiguousarray(site_type, dtype=np.int32)
    st_dev = torch.from_numpy(st).to(dev)
    if centres is None:
        centres = xyz.detach().mean(dim=1)
    sr = None if self_res is None else torch.as_tensor(self_res, dtype=torch.int32, device=dev).contiguous()
    return PoseEnergy.apply(xyz.to(torch.float32), q.to(torch.float32), ff.to(torch.float32),
                            centres.detach().to(torch.float32), engine, int(rep), st, st_dev, sr)


def quat_to_matrix(q):
    """Rotation matrices [..., 3, 3] of quaternions q [..., 4] = (w, x, y, z),
    normalised first (so gradients are tangent to the unit sphere)."""
    return _unit_matrix(q / q.norm(dim=-1, keepdim=True))


def _unit_matrix(q):
    w, x, y, z = q.unbind(-1)
    return torch.stack([
        torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)], -1),
        torch.stack([2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)], -1),
        torch.stack([2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1),
    ], -2)


def _sites_expression(com, quat, tpl):
    return com[:, None, :] + torch.einsum("pij,sj->psi", quat_to_matrix(quat), tpl)


def _plain_cuda(com, quat, tpl):
    """Whether :class:`RigidSites` may take these inputs: dense tensors of one floating type on
    the current GPU, no broadcasting, no gradient of the template, and nothing that has to see the
    tensor operations themselves (tracing or compiling, function transforms, forward-mode
    differentiation, dispatch modes, autocast).  Fewer than 8 poses or one site keep the expression:
    the library's product of such narrow matrices adds its three terms in another order, and the
    single-precision sites would differ in the last bit (equal for all of 8 to 8192 poses tried)."""
    return (_plain(com, quat) and type(tpl) is torch.Tensor and tpl.device == com.device
            and com.dim() == 2 and quat.dim() == 2 and com.shape == (quat.shape[0], 3) and quat.shape[1] == 4
            and com.shape[0] >= 8 and tpl.shape[0] >= 2
            and not (tpl.requires_grad or tpl.is_neg()))


def _torch_hooks():
    """torch's functions that say whether something has to see the tensor operations themselves, or
    None where this torch lacks one of them: the tensor expressions then serve every call."""
    try:
        torch.autograd.forward_ad._current_level
        return (torch._C._functorch.peek_interpreter_stack,
                torch.utils._python_dispatch._get_current_dispatch_mode, torch.compiler.is_compiling,
                torch._C._has_storage)
    except AttributeError:
        return None


_HOOKS = _torch_hooks()


def _watched():
    if _HOOKS is None:
        return True
    transforms, dispatch_mode, compiling, _ = _HOOKS
    # (a compiler must not meet anything but the first question)
    return (compiling() or torch.is_autocast_enabled() or torch.jit.is_tracing() or transforms() is not None
            or torch.autograd.forward_ad._current_level >= 0 or dispatch_mode() is not None)


def _plain(a, b):
    """Two dense tensors of one floating type on the current GPU, and nothing that has to see the
    tensor operations on them."""
    return (not _watched() and type(a) in _TENSORS and type(b) in _TENSORS and a.is_cuda
            and a.dtype in (torch.float32, torch.float64) and b.dtype == a.dtype and b.device == a.device
            and a.device.index == torch.cuda.current_device()
            and not (a.is_neg() or b.is_neg()))


_TENSORS = (torch.Tensor, torch.nn.Parameter)


def _expression_backward(g):
    """Whether a backward pass has to be the tensor expression's: it is to be differentiated
    (create_graph), or runs for a batch of gradients at once (is_grads_batched, vmap)."""
    return torch.is_grad_enabled() or not _HOOKS[3](g)


def _grad_of(expression, inputs, g):
    again = torch.is_grad_enabled()
    with torch.enable_grad():
        return torch.autograd.grad(expression(), inputs, g, create_graph=again)


class RigidSites(torch.autograd.Function):
    """x [P, ns, 3] = com + R(quat / |quat|) t: one kernel each way instead of the
    tensor expression's hundred launches (whose operations it repeats, rounding by rounding).
    Differentiated twice, its backward is the tensor expression's."""

    @staticmethod
    def forward(ctx, com, quat, tpl):
        norm = quat.norm(dim=-1, keepdim=True)
        com_c, unit, tpl = com.contiguous(), (quat / norm).contiguous(), tpl.contiguous()
        P, ns = unit.shape[0], tpl.shape[0]
        out = torch.empty((P, ns, 3), dtype=com.dtype, device=com.device)
        check(lib().gcmc_rigid_sites(int(com.dtype == torch.float64), _p(com_c), _p(unit), _p(tpl), P, ns, _p(out),
                                     _stream()), "gcmc_rigid_sites")
        # (no gradient needs com, and the centres' needs none of the others: those may change)
        ctx.save_for_backward(*((quat, tpl, unit, norm) if ctx.needs_input_grad[1] else ()))
        return out

    @staticmethod
    def backward(ctx, g):
        if not ctx.needs_input_grad[1]:
            return g.sum(1), None, None
        quat, tpl, unit, norm = ctx.saved_tensors
        if _expression_backward(g):
            c = torch.zeros_like(quat[:, :3], requires_grad=True)
            return (*_grad_of(lambda: _sites_expression(c, quat, tpl), (c, quat), g), None)
        g = _dense(g)
        P, ns = g.shape[0], g.shape[1]
        gcom, gquat = unit.new_empty((P, 3)), torch.empty_like(unit)
        check(lib().gcmc_rigid_sites_grad(int(g.dtype == torch.float64), _p(unit), _p(norm), _p(tpl), _p(g), P, ns,
                                          _p(gcom), _p(gquat), _stream()), "gcmc_rigid_sites_grad")
        return gcom, gquat, None


def lj_table(eps_kcal, rmin_half, n_rows: int):
    """Pair table (sigma [nm], eps [kJ/mol]) [n_rows * n * 2] from per-type
    CHARMM eps [kcal/mol] and rmin/2 [A] (n types, the first n_rows being the
    fragment site types): sigma = 2 rmin/2 / 2^(1/6) / 10, eps_kJ = 4.184 eps,
    Lorentz-Berthelot combining (gcmc/python/simulation.py:64-72)."""
    if isinstance(n_rows, (int, np.integer)) and _plain(eps_kcal, rmin_half) and eps_kcal.dim() == 1 \
            and eps_kcal.shape == rmin_half.shape and 1 <= n_rows <= eps_kcal.shape[0] <= 32768:
        # (a copy to save: the caller may change eps between the passes, as with the expression)
        return LJPairs.apply(eps_kcal.clone(), rmin_half, int(n_rows))
    return _lj_expression(eps_kcal, rmin_half, n_rows)


def _lj_expression(eps_kcal, rmin_half, n_rows):
    sigma = 2.0 * rmin_half / 2.0 ** (1.0 / 6.0) / 10.0
    e = V.KCAL_TO_KJ * eps_kcal
    s2 = (sigma[:n_rows, None] + sigma[None, :]) / 2
    e2 = torch.sqrt(e[:n_rows, None] * e[None, :])
    return torch.stack([s2, e2], -1).reshape(-1)


class LJPairs(torch.autograd.Function):
    """The table of :func:`lj_table` by one kernel each way (the tensor expression's operations,
    rounding by rounding: equal for every table of 1 to 59 types tried, both precisions), in place
    of some 35 launches: 950 -> 635 us a pass of 4096 poses with gradients; differentiated twice, its backward is the expression's."""

    @staticmethod
    def forward(ctx, eps, rmin, rows):
        e, r = eps.contiguous(), rmin.contiguous()
        n = e.shape[0]
        out = torch.empty(rows * n * 2, dtype=e.dtype, device=e.device)
        check(lib().gcmc_lj_pairs(int(e.dtype == torch.float64), _p(e), _p(r), n, rows, _p(out), _stream()),
              "gcmc_lj_pairs")
        ctx.save_for_backward(eps)  # (the table is linear in rmin)
        ctx.rows = rows
        return out

    @staticmethod
    def backward(ctx, g):
        (eps,) = ctx.saved_tensors
        if _expression_backward(g):
            e = eps if eps.requires_grad else eps.detach().requires_grad_()
            r = torch.zeros_like(eps, requires_grad=True)
            return (*_grad_of(lambda: _lj_expression(e, r, ctx.rows), (e, r), g), None)
        e, g = eps.contiguous(), _dense(g)
        geps, grmin = torch.empty_like(e), torch.empty_like(e)
        check(lib().gcmc_lj_pairs_grad(int(e.dtype == torch.float64), _p(e), _p(g), e.shape[0], ctx.rows, _p(geps),
                                       _p(grmin), _stream()), "gcmc_lj_pairs_grad")
        return geps, grmin, None


class RigidFragment:
    """Poses of fragment type ``ftype`` of replica ``rep`` of an Engine:
    x_s = com + R(quat) (t_s - mean t)."""

    def __init__(self, engine, rep: int, ftype: int, device="cuda", dtype=torch.float64):
        from . import poses as PZ
        tpl, q, t = PZ.template(engine.systems[rep], ftype)
        self.engine, self.rep, self.ftype = engine, rep, ftype
        self.template = torch.as_tensor(tpl, dtype=dtype, device=device)
        self.charges = torch.as_tensor(q, dtype=dtype, device=device)
        self.site_type = t

    def sites(self, com, quat):
        tpl = self.template.to(com.dtype)
        if _plain_cuda(com, quat, tpl):
            return RigidSites.apply(com, quat, tpl)
        return _sites_expression(com, quat, tpl)

    def energy(self, com, quat, ff, charges=None):
        q = self.charges if charges is None else charges
        return pose_energy(self.engine, self.rep, self.sites(com, quat), q, ff, self.site_type,
                           centres=com.detach())
