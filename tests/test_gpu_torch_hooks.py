"""The differentiable pose energy on a torch without some of the private names it asks (needs a B200)."""
import importlib.util

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("holder,name", [(torch._C._functorch, "peek_interpreter_stack"),
                                         (torch.autograd.forward_ad, "_current_level"),
                                         (torch.utils._python_dispatch, "_get_current_dispatch_mode"),
                                         (torch._C, "_has_storage"), (None, None)])
def test_missing_names_mean_the_expression(monkeypatch, holder, name):
    """Sites and pair table of CUDA tensors, and their gradients, are the tensor expressions' then."""
    import pygcmc_b200.grad as installed
    g = torch.Generator().manual_seed(5)
    com, quat, tpl, w = (torch.randn(s, generator=g, dtype=torch.float64).cuda()
                         for s in ((12, 3), (12, 4), (5, 3), (12, 5, 3)))
    par = [0.1 + torch.rand(9, generator=g, dtype=torch.float64).cuda() for _ in range(2)]
    spec = importlib.util.spec_from_file_location("pygcmc_b200.grad_on_another_torch", installed.__file__)
    grad = importlib.util.module_from_spec(spec)
    frag = type("Frag", (), {"template": tpl})

    def results(sites, table):
        leaves = [v.clone().requires_grad_() for v in (com, quat, *par)]
        x, y = sites(leaves[0], leaves[1]), table(leaves[2], leaves[3])
        node = type(x.grad_fn).__name__, type(y.grad_fn).__name__
        return node, [x, y, *torch.autograd.grad((x * w).sum() + (y * y).sum(), leaves)]
    want = results(lambda c, q: installed._sites_expression(c, q, tpl), lambda e, r: installed._lj_expression(e, r, 4))
    with monkeypatch.context() as m:
        if holder is not None:
            m.delattr(holder, name)
        spec.loader.exec_module(grad)
        node, got = results(lambda c, q: grad.RigidFragment.sites(frag, c, q), lambda e, r: grad.lj_table(e, r, 4))
    fused = node == ("RigidSitesBackward", "LJPairsBackward")
    assert fused == (holder is None), node
    for a, b in zip(got, want[1]):
        assert torch.allclose(a, b, rtol=1e-11, atol=1e-11)


@pytest.mark.parametrize("backend", ["eager", "aot_eager"])
def test_compiled_whole(backend):
    """Under a compiler that allows no break in the graph the sites and the pair table are the expressions, with
    their gradients."""
    import pygcmc_b200.grad as grad
    g = torch.Generator().manual_seed(6)
    com, quat, tpl = (torch.randn(s, generator=g, dtype=torch.float64).cuda() for s in ((16, 3), (16, 4), (5, 3)))
    par = [0.1 + torch.rand(9, generator=g, dtype=torch.float64).cuda() for _ in range(2)]
    frag = type("Frag", (), {"template": tpl})
    for f, ref, inputs in (
            (lambda c, q: grad.RigidFragment.sites(frag, c, q), lambda c, q: grad._sites_expression(c, q, tpl),
             (com, quat)),
            (lambda e, r: grad.lj_table(e, r, 4), lambda e, r: grad._lj_expression(e, r, 4), par)):
        got = []
        for fn in (torch.compile(f, backend=backend, fullgraph=True), ref):
            leaves = [v.clone().requires_grad_() for v in inputs]
            out = fn(*leaves)
            got.append([out, *torch.autograd.grad((out * out).sum(), leaves)])
        for a, b in zip(*got):
            assert torch.allclose(a, b, rtol=1e-11, atol=1e-11)
