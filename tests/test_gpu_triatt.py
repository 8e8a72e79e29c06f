"""Triangle attention on the GPU against the CPU oracle.  The reference has no such op, so there are no
golden vectors from it: parity is against the oracle's fp64 statement of the algorithm, plus the
masking / padding invariances the reference tests for its own pair ops."""
import pytest
import torch

import helpers as H
from gpu_util import assert_close
from oracle import pair_ops as O

pytestmark = pytest.mark.gpu


def _module(w: dict, ending: bool):
    import bioemu2_b200 as b

    m = b.TriangleAttention(ending=ending).eval()
    m.load_state_dict(w, strict=True)
    return m.cuda()


@pytest.mark.parametrize("ending", [False, True])
@pytest.mark.parametrize("N,dtype", [(24, torch.float32), (128, torch.float32), (200, torch.bfloat16), (129, torch.float32)])
def test_triatt_vs_oracle(ending, N, dtype):
    g = torch.Generator().manual_seed(500 + N)
    w = H.triatt_weights(g)
    x = torch.randn(1, N, N, 128, generator=g).to(dtype)
    mask = torch.rand(1, N, N, generator=g) > 0.2
    ref = O.triangle_attention(x.double(), mask, {k: v.double() for k, v in w.items()}, 4, ending)
    m = _module(w, ending)
    with torch.no_grad():
        out = m(x.cuda(), mask.cuda())
    assert out.dtype == dtype
    assert_close(f"triatt_{'end' if ending else 'start'}_N{N}_{dtype}", out, ref)


@pytest.mark.parametrize("ending", [False, True])
@pytest.mark.parametrize("N,dtype", [(131, torch.float32), (160, torch.bfloat16), (192, torch.float32), (319, torch.bfloat16)])
def test_lines_of_an_odd_number_of_half_tiles(ending, N, dtype):
    """Projection tiles that hold the end of one line and the start of the next, the last without a second half (131, 319); in place
    the result is the update added, with a rounding of the update in `out` and one of the sum."""
    g = torch.Generator().manual_seed(800 + N)
    w = H.triatt_weights(g)
    x = torch.randn(1, N, N, 128, generator=g).to(dtype)
    mask = torch.rand(1, N, N, generator=g) > 0.2
    ref = O.triangle_attention(x.double(), mask, {k: v.double() for k, v in w.items()}, 4, ending)
    m = _module(w, ending)
    with torch.no_grad():
        out = m(x.cuda(), mask.cuda())
        z = x.cuda()
        m.forward_residual_(z, mask.cuda())
    assert_close(f"half_tiles_{'end' if ending else 'start'}_N{N}_{dtype}", out, ref)
    bound = 1.5 * torch.finfo(dtype).eps * (x.cuda().float().abs() + out.float().abs()) + 1e-6
    assert ((z.float() - (x.cuda().float() + out.float())).abs() <= bound).all()


@pytest.mark.parametrize("ending", [False, True])
def test_triatt_residual_inplace_and_padding(ending):
    N, P = 70, 6
    g = torch.Generator().manual_seed(77)
    w = H.triatt_weights(g)
    x = torch.randn(2, N, N, 128, generator=g)
    tok = torch.ones(2, N, dtype=torch.bool)
    tok[0, N - 4:] = False
    mask = tok[:, :, None] & tok[:, None, :]
    m = _module(w, ending)
    with torch.no_grad():
        upd = m(x.cuda(), mask.cuda())
        z = x.cuda().clone()
        ret = m.forward_residual_(z, mask.cuda())
        assert ret.data_ptr() == z.data_ptr()
        torch.testing.assert_close(z, x.cuda() + upd, atol=1e-5, rtol=1e-5)
        xp = torch.full((2, N + P, N + P, 128), 1000.0)
        xp[:, :N, :N] = x
        mp = torch.zeros(2, N + P, N + P, dtype=torch.bool)
        mp[:, :N, :N] = mask
        upd_p = m(xp.cuda(), mp.cuda())[:, :N, :N]
    valid = (tok[:, :, None] & tok[:, None, :]).cuda()
    torch.testing.assert_close(upd_p[valid], upd[valid], atol=2e-3, rtol=0)


@pytest.mark.parametrize("N,B", [(1, 1), (7, 2), (63, 1), (64, 1), (65, 1), (100, 2), (127, 1), (128, 1), (129, 1)])
@pytest.mark.parametrize("ending", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("scale", [1.0, 60.0])
def test_short_lines_in_place_are_the_update_added(N, B, ending, dtype, scale):
    """Lines of up to 128 positions are attended to and projected in one kernel when the update is added in place: the same bits as the
    update by itself, added in fp32 (one rounding of the sum in bf16).  Masks with padding, holes and lines without a valid key;
    logits in the range of a row's reference and far outside it."""
    import bioemu2_b200 as b
    from bioemu2_b200 import _lib

    g = torch.Generator(device="cuda").manual_seed(3000 + N)
    with torch.device("cuda"):
        m = b.TriangleAttention(ending=ending).eval()
    with torch.no_grad():
        for name, p in m.named_parameters():
            if p.ndim >= 2:
                p.uniform_(-128 ** -0.5, 128 ** -0.5, generator=g)
        m.linear_b.weight.mul_(scale)
        z = torch.randn(B, N, N, 128, device="cuda", generator=g).to(dtype)
        mask = torch.rand(B, N, N, device="cuda", generator=g) > 0.2
        mask[:, :, N - N // 4:] = False
        mask[:, :, N // 3:N // 2] = False
        mask[:, N - N // 5:] = False
        mask[:, :1] = True
        want = z.float() + m(z, mask).float()
        got = z.clone()
        m.forward_residual_(got, mask)
    assert _lib.device_status() == 0
    if dtype == torch.float32:
        assert torch.equal(got, want)
    else:
        torch.testing.assert_close(got.float(), want, rtol=2 ** -8, atol=2 ** -9 * want.abs().max().item())


@pytest.mark.parametrize("N,B,ending", [(1, 1, True), (24, 1, False), (65, 2, True), (100, 1, True), (128, 1, False), (128, 1, True),
                                        (129, 1, True), (150, 2, True), (203, 1, True), (300, 1, True)])
def test_bf16_update_added_in_place_is_rounded_once(N, B, ending):
    """Short lines, and ending-node lines that are not whole tiles of 128: the bf16 result is the rounding of what the same rows
    give in fp32 (the projection's fp32 result rounded to bf16 before the sum would be off in 3 % to 7 % of the values)."""
    import bioemu2_b200 as b
    from bioemu2_b200 import _lib

    g = torch.Generator(device="cuda").manual_seed(3300 + N)
    with torch.device("cuda"):
        m = b.TriangleAttention(ending=ending).eval()
    with torch.no_grad():
        for p in m.parameters():
            if p.ndim >= 2:
                p.uniform_(-128 ** -0.5, 128 ** -0.5, generator=g)
        z = torch.randn(B, N, N, 128, device="cuda", generator=g).bfloat16()
        mask = torch.rand(B, N, N, device="cuda", generator=g) > 0.2
        want = m.forward_residual_(z.float(), mask).bfloat16()
        got = m.forward_residual_(z.clone(), mask)
    assert _lib.device_status() == 0
    assert torch.equal(got, want)
