"""The native accurate triangle multiplication and transition against fp64, at token counts around their 8-, 32- and 128-wide
pieces and at widths on either side of the native transition's rule (multiples of 64)."""
import pytest
import torch
import torch.nn.functional as TF

pytestmark = pytest.mark.gpu


def _rel(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


def _module(m, seed):
    g = torch.Generator().manual_seed(seed)
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (p.shape[-1] ** -0.5 if p.ndim == 2 else 0.2) + (p.ndim == 1))
    return m.eval().cuda()


@pytest.mark.parametrize("mode", ["outgoing", "incoming"])
@pytest.mark.parametrize("n", [1, 8, 13, 33, 129])
def test_triangle_multiplication(n, mode):
    import bioemu2_b200 as b

    m = _module(b.TriangleMultiplication(128, mode, matmul_precision="ieee"), n)
    x = torch.randn(2, n, n, 128, device="cuda")
    mask = torch.rand(2, n, n, device="cuda") > 0.2
    mask[:, 0, 0] = True
    with torch.no_grad():
        got = m(x, mask)
        inplace = m.forward_residual_(x.clone(), mask)
        w = {k: v.double() for k, v in m.state_dict().items()}
        h = TF.layer_norm(x.double(), (128,), w["norm_in.weight"], w["norm_in.bias"])
        ab = (h @ w["p_in.weight"].T) * torch.sigmoid(h @ w["g_in.weight"].T) * mask[..., None]
        eq = "bikd,bjkd->bijd" if mode == "outgoing" else "bkid,bkjd->bijd"
        t = TF.layer_norm(torch.einsum(eq, ab[..., :128], ab[..., 128:]), (128,), w["norm_out.weight"], w["norm_out.bias"])
        want = (t @ w["p_out.weight"].T) * torch.sigmoid(h @ w["g_out.weight"].T)
    assert _rel(got, want) < 5e-5
    torch.testing.assert_close(inplace, x + got, atol=1e-6, rtol=1e-6)


@pytest.mark.parametrize("rows,dim,hidden,out", [(1, 128, 512, 128), (131, 128, 64, 128), (130, 192, 320, 192), (77, 64, 192, 40),
                                                 (50, 128, 72, 128), (33, 72, 128, 72)])
@pytest.mark.parametrize("norm", [True, False])
def test_transition(rows, dim, hidden, out, norm):
    import bioemu2_b200 as b

    m = _module(b.Transition(dim, hidden, out, use_norm=norm), rows)
    x = torch.randn(rows, dim, device="cuda")
    with torch.no_grad(), b.precision.matmul_precision("ieee"):
        got = m(x)
        w = {k: v.double() for k, v in m.state_dict().items()}
        h = TF.layer_norm(x.double(), (dim,), w["norm.weight"], w["norm.bias"]) if norm else x.double()
        want = (TF.silu(h @ w["fc1.weight"].T) * (h @ w["fc2.weight"].T)) @ w["fc3.weight"].T
        assert _rel(got, want) < 5e-5
        if out == dim:
            torch.testing.assert_close(m.forward_residual_(x.clone()), x + got, atol=1e-5, rtol=1e-5)


def test_swiglu_keeps_fp32_where_the_gate_is_nearly_shut():
    """silu(a) * b far below zero, where an exponential whose argument is rounded to a multiple of 2^-17 shows.  What the output
    keeps of a value is its (hi | lo): lo is at most half a unit of hi's eighth bit and is rounded to eight bits itself, 2^-17
    of the value at the most and, over evenly spread significands, 0.32 * 2^-17 = 2.4e-6 in the root mean square."""
    import bioemu2_b200 as b

    rows = 4096
    m = b.Transition(128, 64, 64, use_norm=False).eval().cuda()
    with torch.no_grad():
        for p in m.parameters():
            p.zero_()
        m.fc1.weight[:, 0] = 1.0
        m.fc2.weight[:, 1] = 1.0
        m.fc3.weight.copy_(torch.eye(64))
    g = torch.Generator().manual_seed(61)
    a = (-40.0 - 40.0 * torch.rand(rows, generator=g)).cuda()
    hi = a.bfloat16()
    a = hi.float() + (a - hi.float()).bfloat16().float()  # what the product's split operands hold
    x = torch.zeros(rows + 5, 128, device="cuda")
    x[:rows, 0], x[:, 1] = a, 2.0 ** 60
    x[rows:, 0] = torch.tensor([-88.0, -89.0, -3.0e5, 0.0, float("nan")])
    x[rows + 3, 1] = 3.0
    with torch.no_grad(), b.precision.matmul_precision("ieee"):
        got = m(x).double()
    assert torch.equal(got[:-1, :1].expand(-1, 64), got[:-1])
    want = a.double() * torch.sigmoid(a.double()) * 2.0 ** 60
    rel = (got[:rows, 0] - want) / want
    assert rel.abs().max() <= 2.0 ** -17 + 2.0 ** -21
    assert rel.square().mean().sqrt() < 2.6e-6
    assert got[rows, 0] != 0 and not got[rows + 1:rows + 4].any() and not torch.isnan(got[:-1]).any() and torch.isnan(got[-1]).all()
