"""The fused rigid-site and pair-table kernels against the tensor expressions they stand for (needs a B200).

Forward: every operation is rounded alike and a matrix product's three terms are a fused
multiply-add chain, so the sites agree to the last bit or, should the library's product order its
terms differently, to a rounding of the largest term: 4 eps (|com| + |t|).  Backward: sums of ns
products, FP64 inside: ns eps of the sum of |terms| plus the expression's own rounding, 64 eps of
that sum in all.  Inputs that the fused path does not take, and second derivatives, follow the
expression.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def inputs(P, ns, dtype, seed=0):
    g = torch.Generator().manual_seed(seed + 31 * P + ns)
    com = 60 * torch.rand((P, 3), generator=g, dtype=torch.float64)
    quat = torch.randn((P, 4), generator=g, dtype=torch.float64)
    tpl = 2 * torch.randn((ns, 3), generator=g, dtype=torch.float64)
    w = torch.randn((P, ns, 3), generator=g, dtype=torch.float64)
    return [t.to("cuda", dtype) for t in (com, quat, tpl, w)]


class Frag:
    def __init__(self, tpl):
        self.template = tpl


def fused(com, quat, tpl):
    from pygcmc_b200.grad import RigidFragment
    return RigidFragment.sites(Frag(tpl), com, quat)


def expression(com, quat, tpl):
    from pygcmc_b200.grad import quat_to_matrix
    return com[:, None, :] + torch.einsum("pij,sj->psi", quat_to_matrix(quat), tpl)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("P,ns", [(1, 1), (7, 3), (8, 2), (61, 3), (63, 20), (64, 4), (65, 12), (1000, 7), (4096, 5)])
def test_sites_and_gradients(P, ns, dtype):
    com, quat, tpl, w = inputs(P, ns, dtype)
    eps = torch.finfo(dtype).eps
    c, q = com.clone().requires_grad_(), quat.clone().requires_grad_()
    x = fused(c, q, tpl)
    assert (type(x.grad_fn).__name__ == "RigidSitesBackward") == (P >= 8 and ns >= 2)
    ref = expression(com, quat, tpl)
    bound = 4 * eps * (com.abs().amax() + tpl.abs().amax())
    assert (x - ref).abs().max() <= bound
    (x * w).sum().backward()
    c2, q2 = (t.double().clone().requires_grad_() for t in (com, quat))
    (expression(c2, q2, tpl.double()) * w.double()).sum().backward()
    l1c = w.double().abs().sum(1)
    l1q = (w.double().abs().sum(2) @ tpl.double().abs().sum(1, keepdim=True)) * 8 / quat.double().norm(dim=1)[:, None]
    assert ((c.grad.double() - c2.grad).abs() <= 64 * eps * l1c).all()
    assert ((q.grad.double() - q2.grad).abs() <= 64 * eps * l1q).all()


def test_forms_outside_the_fused_path():
    com, quat, tpl, w = inputs(33, 6, torch.float64)
    ref = expression(com, quat, tpl)
    # strided inputs (fused), one quaternion for all poses, mixed types, a differentiable template, the CPU
    buf = torch.zeros((33, 8), device="cuda", dtype=torch.float64)
    buf[:, ::2] = quat
    assert torch.allclose(fused(com.t().contiguous().t(), buf[:, ::2], tpl), ref, rtol=0, atol=1e-13)
    assert torch.allclose(fused(com, quat[:1], tpl), expression(com, quat[:1], tpl), rtol=0, atol=1e-13)
    t = tpl.clone().requires_grad_()
    fused(com, quat, t).sum().backward()
    assert t.grad is not None
    assert torch.allclose(fused(com.cpu(), quat.cpu(), tpl.cpu()).cuda(), ref, rtol=0, atol=1e-13)
    assert fused(com[:0], quat[:0], tpl).shape == (0, 6, 3)
    assert torch.allclose(fused(torch._neg_view(-com), quat, tpl), ref, rtol=0, atol=1e-13)
    # the table: the rows given as None (all of them) or as a float (refused)
    from pygcmc_b200.grad import _lj_expression, lj_table
    e, r = quat[:, 0].abs(), quat[:, 1].abs()
    assert torch.equal(lj_table(e, r, None), _lj_expression(e, r, None))
    assert torch.equal(lj_table(torch._neg_view(-e), r, 5), _lj_expression(e, r, 5))
    with pytest.raises(TypeError):
        lj_table(e, r, 5.0)
    # function transforms and forward mode
    one = torch.func.vmap(lambda c, q: expression(c[None], q[None], tpl)[0])(com, quat)
    assert torch.allclose(torch.func.vmap(lambda c, q: fused(c[None], q[None], tpl)[0])(com, quat), one, rtol=0,
                          atol=1e-13)
    _, jv = torch.func.jvp(lambda q: fused(com, q, tpl), (quat,), (quat + 1,))
    _, jr = torch.func.jvp(lambda q: expression(com, q, tpl), (quat,), (quat + 1,))
    assert torch.allclose(jv, jr, rtol=1e-12, atol=1e-12)
    # second derivatives
    q = quat.clone().requires_grad_()
    for f in (fused, expression):
        (g,) = torch.autograd.grad((f(com, q, tpl) * w).sum(), q, create_graph=True)
        (h,) = torch.autograd.grad((g * g).sum(), q)
        if f is fused:
            first = h
    assert torch.allclose(first, h, rtol=1e-10, atol=1e-10)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n,rows", [(1, 1), (2, 1), (24, 23), (31, 31), (33, 32), (70, 40)])
def test_pair_table(n, rows, dtype):
    """Values: the same roundings, so equal to the last bit or at most one of them (4 eps); gradients:
    sums of at most n + rows terms, 64 eps of the sum of |terms|."""
    from pygcmc_b200.grad import _lj_expression, lj_table
    g = torch.Generator().manual_seed(n)
    eps = (0.02 + 0.18 * torch.rand(n, generator=g, dtype=torch.float64)).to("cuda", dtype)
    rmin = (1.0 + 1.2 * torch.rand(n, generator=g, dtype=torch.float64)).to("cuda", dtype)
    w = torch.randn(rows * n * 2, generator=g, dtype=torch.float64).to("cuda", dtype)
    e, r = eps.clone().requires_grad_(), rmin.clone().requires_grad_()
    out = lj_table(e, r, rows)
    assert type(out.grad_fn).__name__ == "LJPairsBackward"
    u = torch.finfo(dtype).eps
    ref = _lj_expression(eps, rmin, rows)
    assert ((out - ref).abs() <= 4 * u * ref.abs()).all()
    (out * w).sum().backward()
    want = []
    for weights in (w.double(), w.double().abs()):  # the gradients, and the sums of |terms|
        e2, r2 = (t.detach().double().clone().requires_grad_() for t in (eps, rmin))
        (_lj_expression(e2, r2, rows) * weights).sum().backward()
        want.append((e2.grad, r2.grad))
    for got, exact, scale in zip((e.grad, r.grad), *want):
        assert ((got.double() - exact).abs() <= 64 * u * scale).all()
    # another type of the parameters, and second derivatives, follow the expression
    assert torch.allclose(lj_table(eps.double(), rmin.float(), rows).double(), ref.double(), rtol=1e-6)
    e3 = eps.clone().requires_grad_()
    hs = []
    for f in (lj_table, _lj_expression):
        (d,) = torch.autograd.grad((f(e3, rmin, rows) * w).sum(), e3, create_graph=True)
        (h,) = torch.autograd.grad((d * d).sum(), e3)
        hs.append(h)
    assert torch.allclose(*hs, rtol=1e-3 if dtype == torch.float32 else 1e-10)


@pytest.mark.parametrize("P,ns,nff", [(1, 1, 2), (0, 3, 0), (85, 3, 7), (86, 1, 256), (255, 20, 257), (4097, 5, 1104)])
def test_chain_rule_of_pose_gradients(P, ns, nff):
    """Products and conversions are single roundings (equal); the sum over the poses in FP64 and one
    rounding to FP32: 2^-24 of the sum and P 2^-53 of the sum of |terms|."""
    import ctypes
    from pygcmc_b200._native import check, lib
    g = torch.Generator().manual_seed(P + ns)
    w, gx, gq, gff = (torch.randn(s, generator=g, dtype=torch.float64).cuda() for s in ((P,), (P, ns, 3), (P, ns), (nff,)))
    out = [torch.full(s, 7.0, device="cuda") for s in ((P, ns, 3), (ns,), (nff,))]

    def p(t):
        return ctypes.c_void_p(t.data_ptr())
    stream = ctypes.c_void_p(1)
    check(lib().gcmc_pose_chain(p(w), p(gx), p(gq), p(gff), P, ns, nff, *map(p, out), stream), "gcmc_pose_chain")
    want = (gq * w[:, None]).sum(0)
    assert torch.equal(out[0], (gx * w[:, None, None]).float())
    assert torch.equal(out[2], gff.float())
    assert ((out[1].double() - want).abs() <= 2.0 ** -23 * want.abs() + P * 2.0 ** -52 * (gq * w[:, None]).abs().sum(0)).all()
    kept = out[1].clone()  # the charges' sum alone, again: the same bits
    out[1].zero_()
    check(lib().gcmc_pose_chain(p(w), None, p(gq), None, P, ns, 0, None, p(out[1]), None, stream), "gcmc_pose_chain")
    assert torch.equal(out[1], kept)


def test_inputs_may_change_before_the_backward():
    """Centres and the table's parameters are not needed by any gradient as they stand: in-place updates
    between the two passes are allowed, as with the expressions."""
    from pygcmc_b200.grad import _lj_expression, lj_table
    com, quat, tpl, w = inputs(40, 5, torch.float64)
    eps, rmin = com[:, 0].abs() + 0.1, quat[:, 0].abs() + 1
    got = []
    for sites, table in ((fused, lj_table), (expression, _lj_expression)):
        c, q, e, r = (t.clone().requires_grad_() for t in (com, quat, eps, rmin))
        out = (sites(c, q, tpl) * w).sum() + (table(e, r, 7) ** 2).sum()
        with torch.no_grad():
            for t in (c, e, r):
                t += 1
        out.backward()
        got.append((c.grad, q.grad, e.grad, r.grad))
    for a, b in zip(*got):
        assert torch.allclose(a, b, rtol=1e-11, atol=1e-11)


def test_batched_gradients():
    """Several output gradients at once (is_grads_batched) give what the expressions give."""
    from pygcmc_b200.grad import _lj_expression, lj_table
    com, quat, tpl, w = inputs(12, 4, torch.float64)
    eps, rmin = com[:, 0].abs() + 0.1, quat[:, 0].abs() + 1
    got = []
    for sites, table in ((fused, lj_table), (expression, _lj_expression)):
        c, q, e, r = (t.clone().requires_grad_() for t in (com, quat, eps, rmin))
        x, y = sites(c, q, tpl), table(e, r, 7)
        many = torch.stack([w, 2 * w, w.flip(0)])
        got.append(torch.autograd.grad(x, (c, q), many, is_grads_batched=True)
                   + torch.autograd.grad(y, (e, r), many.reshape(3, -1)[:, :1].expand(3, y.numel()), is_grads_batched=True))
    for a, b in zip(*got):
        assert torch.allclose(a, b, rtol=1e-11, atol=1e-11)
