"""What the fused rigid sites keep between the passes (needs a B200)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


class Frag:
    def __init__(self, tpl):
        self.template = tpl


def expression(com, quat, tpl):
    from pygcmc_b200.grad import quat_to_matrix
    return com[:, None, :] + torch.einsum("pij,sj->psi", quat_to_matrix(quat), tpl)


@pytest.mark.parametrize("needs", ["com", "quat", "both"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_only_what_a_gradient_needs_is_kept(needs, dtype):
    """As with the tensor expression: inputs that no requested gradient uses may change between the passes, the
    others are refused then, and the gradients, first and batched and of a second differentiation, are the
    expression's (sums of 5 terms and of the rotation's: 64 eps of their magnitude, below 200)."""
    from pygcmc_b200.grad import RigidFragment
    g = torch.Generator().manual_seed(3)
    com, quat, tpl, w = (torch.randn(s, generator=g, dtype=torch.float64).to("cuda", dtype)
                         for s in ((40, 3), (40, 4), (5, 3), (40, 5, 3)))
    tol = 64 * torch.finfo(dtype).eps * 200
    got = []
    for sites in (lambda c, q, t: RigidFragment.sites(Frag(t), c, q), expression):
        c, q, t = com.clone(), quat.clone(), tpl.clone()
        wanted = [v.requires_grad_() for v, name in ((c, "com"), (q, "quat")) if needs in (name, "both")]
        x = sites(c, q, t)
        many = torch.autograd.grad(x, wanted, torch.stack([w, 2 * w]), is_grads_batched=True, retain_graph=True)
        again = torch.autograd.grad(x, wanted, w, create_graph=True)
        refused = []
        for v in (c, q, t):
            if v is t or needs == "com" or v is c:
                with torch.no_grad():
                    v.add_(1)
            try:
                first = torch.autograd.grad(x, wanted, w, retain_graph=True)
                refused.append(False)
            except RuntimeError:
                refused.append(True)
        got.append((refused, [*many, *again]))
        if needs == "com":
            assert refused == [False] * 3
            got[-1][1].extend(first)
    assert got[0][0] == got[1][0]
    for a, b in zip(got[0][1], got[1][1]):
        assert (a - b).abs().max() <= tol
