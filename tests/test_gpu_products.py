"""Products with fused epilogues, the kernels around them and the native compositions, at the edges of their tiles, against
plain fp32 arithmetic or the module-by-module path."""
import pytest
import torch
import torch.nn.functional as TF

pytestmark = pytest.mark.gpu
F32, BF16 = torch.float32, torch.bfloat16


def _close(got, want):
    import bioemu2_b200._lib as L

    assert L.device_status() == 0
    d, want = (got.double() - want.double()).abs(), want.double()
    assert d.norm() <= 1e-2 * want.norm() and d.max() <= 2e-2 * want.abs().max()


def _gen(*key):
    return torch.Generator().manual_seed(sum((i + 1) * 7919 * k for i, k in enumerate(key)))


def _fill(m, seed):
    g = _gen(seed)
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (p.shape[-1] ** -0.5 if p.ndim == 2 else 0.2) + (p.ndim == 1))
    return m.eval().cuda()


@pytest.mark.parametrize("rows,n,k", [(1, 8, 8), (127, 120, 72), (129, 136, 64), (300, 264, 320), (1000, 768, 768), (20000, 128, 136)])
@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("residual", [None, "out", "other"])
def test_linear_epilogues(rows, n, k, dtype, residual):
    from bioemu2_b200 import functional as F

    g = _gen(rows, n, k)
    x, w = torch.randn(rows, k, generator=g).to(BF16).cuda(), (torch.randn(n, k, generator=g) * k ** -0.5).to(BF16).cuda()
    bias, r = torch.randn(n, generator=g).cuda(), torch.randn(rows, n, generator=g).to(dtype).cuda()
    want = x.double() @ w.double().T + bias.double() + (r.double() if residual else 0)
    out = r.clone() if residual == "out" else torch.empty(rows, n, dtype=dtype, device="cuda")
    res = out if residual == "out" else r if residual else None
    _close(F.linear_bf16(x, w, bias, res, out_dtype=dtype, out=out), want)


@pytest.mark.parametrize("rows", [1, 127, 129, 20000])
@pytest.mark.parametrize("sources", [1, 2])
@pytest.mark.parametrize("dtype,residual", [(F32, True), (F32, False), (BF16, True)])
def test_ln_linear(rows, sources, dtype, residual):
    from bioemu2_b200 import functional as F

    g = _gen(rows, sources)
    xs = [torch.randn(rows, 128, generator=g).to(dtype).cuda() for _ in range(sources)]
    w = (torch.randn(128, 128 * sources, generator=g) * 0.08).to(BF16).cuda()
    ln_w, ln_b = (torch.randn(128 * sources, generator=g).cuda() for _ in range(2))
    r = torch.randn(rows, 128, generator=g).cuda() if residual else None
    got = F.ln_linear(xs[0], xs[1] if sources == 2 else None, ln_w, ln_b, w, residual=r)
    h = TF.layer_norm(torch.cat(xs, -1).double(), (128 * sources,), ln_w.double(), ln_b.double())
    want = h @ w.double().T + (r.double() if residual else 0)
    _close(got, want)


@pytest.mark.parametrize("rows,dim,hidden", [(1, 128, 256), (130, 128, 200), (19000, 128, 256), (3, 384, 1536), (257, 384, 192),
                                             (257, 384, 200), (140, 72, 64)])
@pytest.mark.parametrize("dtype", [F32, BF16])
def test_transition_widths(rows, dim, hidden, dtype):
    """The fused kernel at 256 hidden units, the general path with its SwiGLU in the product (hidden % 64 == 0) and without."""
    import bioemu2_b200 as b

    m = _fill(b.Transition(dim, hidden), rows + hidden)
    x = torch.randn(rows, dim, generator=_gen(rows, dim)).to(dtype).cuda()
    w = {k: v.double() for k, v in m.state_dict().items()}
    h = TF.layer_norm(x.double(), (dim,), w["norm.weight"], w["norm.bias"])
    want = (TF.silu(h @ w["fc1.weight"].T) * (h @ w["fc2.weight"].T)) @ w["fc3.weight"].T
    with torch.no_grad():
        _close(m(x), want)
        _close(m.forward_residual_(x.clone()), x.double() + want)


@pytest.mark.parametrize("windowed,dim,n,B,M,hidden", [(False, 768, 40, 1, 1, 1536), (False, 384, 136, 2, 3, 768), (False, 96, 136, 1, 2, 192),
                                                       (True, 128, 64, 2, 2, 256), (True, 128, 32, 1, 5, 512), (True, 64, 96, 1, 1, 128)])
@pytest.mark.parametrize("dtype", [F32, BF16])
def test_conditioned_layer_native_against_its_parts(windowed, dim, n, B, M, hidden, dtype):
    import bioemu2_b200 as b

    g = _gen(dim, n, B, M)
    kw = dict(is_sliding_window=True, window_queries=32, window_keys=128) if windowed else {}
    layer = _fill(b.ConditionedTransformerLayer(dim, 16 if windowed else 128, 128, 4 if windowed else dim // 48, hidden, **kw), dim)
    x, c = torch.randn(B * M, n, dim, generator=g).to(dtype).cuda(), torch.randn(B * M, n, 128, generator=g).to(dtype).cuda()
    pairs = torch.randn(*((B, n // 32, 32, 128, 16) if windowed else (B, n, n, 128)), generator=g).to(dtype).cuda()
    mask = (torch.rand(B, n, generator=g) > 0.1).cuda()
    with torch.no_grad():
        assert layer.packed()[2] is not None
        got = layer(x, pairs, c, mask, M)
        want = layer._forward(x, pairs, c, mask, M, layer.attention)
    assert got.dtype == dtype
    _close(got, want)


@pytest.mark.parametrize("n,B,M,hidden,c_dtype,lns", [
    (32, 1, 1, 256, F32, 1.0),      # a quarter of a tile of tokens
    (96, 1, 3, 200, BF16, 0.5),     # two tiles and a part of one, hidden units padded to 256
    (4800, 1, 8, 256, F32, 0.25),   # three tiles for some CTAs
    (2432, 2, 4, 512, BF16, 1.0),   # eight chunks of hidden units, two tiles for some
])
def test_atom_layer_between_its_attention(n, B, M, hidden, c_dtype, lns):
    """The kernels on either side of the window attention at 128 channels, in place and not, against the layer's modules.  Bound: bf16
    operands, as for the other products."""
    import bioemu2_b200 as b
    from bioemu2_b200 import _lib
    from bioemu2_b200 import functional as F

    g = _gen(n, B, M)
    layer = _fill(b.ConditionedTransformerLayer(128, 16, 128, 4, hidden, is_sliding_window=True, window_queries=32, window_keys=128,
                                                lns_scale=lns), n)
    x, c = 3.0 + torch.randn(B * M, n, 128, generator=g).cuda(), torch.randn(B * M, n, 128, generator=g).to(c_dtype).cuda()
    pairs = torch.randn(B, n // 32, 32, 128, 16, generator=g).cuda()
    mask = (torch.rand(B, n, generator=g) > 0.1).cuda()
    kept = x.clone()
    with torch.no_grad():
        got = layer(x, pairs, c, mask, M)
        assert torch.equal(x, kept)
        want = layer._forward(x, pairs, c, mask, M, layer.attention)
        sized = _lib.CondLayer.from_buffer_copy(layer.packed()[2][0])
        sized.B, sized.M, sized.N, sized.lns_scale = B, M, n, lns
        F.cond_layer(sized, x, pairs, None, c, mask, out=x)
    assert _lib.device_status() == 0
    assert torch.equal(x, got)
    _close(got - kept, want - kept)


@pytest.mark.parametrize("S,n,H,c_m", [(1, 1, 1, 8), (3, 37, 8, 64), (5, 130, 6, 64), (2, 264, 16, 72)])
def test_pwa_values(S, n, H, c_m):
    from bioemu2_b200 import functional as F
    from bioemu2_b200._lib import check, lib

    g = _gen(S, n, H)
    pitch = F.pad8(n)
    w, mn = torch.randn(H * 32, c_m, generator=g).to(BF16).cuda(), torch.randn(S, n, c_m, generator=g).to(BF16).cuda()
    vT = torch.full((H, S * 32, pitch), 7.0, dtype=BF16, device="cuda")
    check(lib.b200_pwa_values(w.data_ptr(), mn.data_ptr(), vT.data_ptr(), S, n, c_m, H, pitch, F._stream()))
    want = torch.zeros(H, S, 32, pitch, dtype=torch.float64, device="cuda")
    want[..., :n] = torch.einsum("hdc,sjc->hsdj", w.double().view(H, 32, c_m), mn.double())
    _close(vT, want.view(H, S * 32, pitch))


@pytest.mark.parametrize("B,S,n", [(1, 1, 1), (2, 70, 37), (1, 33, 130)])
def test_outer_product_mean_added_to_the_pair_tensor(B, S, n):
    import bioemu2_b200 as b

    g = _gen(B, S, n)
    mod = _fill(b.OuterProductMean(64, 32, 128), n)
    m, z = torch.randn(B, S, n, 64, generator=g).cuda(), torch.randn(B, n, n, 128, generator=g).cuda()
    mask = (torch.rand(B, S, n, generator=g) > 0.2).cuda()
    with torch.no_grad():
        torch.testing.assert_close(mod.forward_add(m, mask, z), z + mod(m, mask), atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("n,B", [(1, 1), (40, 2), (130, 1)])
def test_trunk_call_against_its_layers(n, B):
    import bioemu2_b200 as b

    g = _gen(n, B)
    trunk = _fill(b.PairformerModule(384, 128, 2), n)
    s, z = torch.randn(B, n, 384, generator=g).cuda(), torch.randn(B, n, n, 128, generator=g).cuda()
    mask = torch.rand(B, n, generator=g) > 0.1
    mask[:, 0] = True
    mask = mask.cuda()
    with torch.no_grad():
        first, again = trunk(s, z, mask), trunk(s, z, mask)  # weights packed block by block under the stack, then kept
        s1, z1 = s, z
        for layer in trunk.layers:
            s1, z1 = layer(s1, z1, mask)
    for got in (first, again):
        _close(got[0], s1)
        _close(got[1], z1)


def test_packed_weights_layout():
    from bioemu2_b200 import functional as F

    g = _gen(3)
    a, c, d = torch.randn(6, 40, generator=g).cuda(), torch.randn(4, 16, generator=g).cuda(), torch.randn(4, 16, generator=g).cuda()
    pk = F._Pack()
    o1 = pk.add(a, scale=0.5, groups=3, pad_to=96)      # 80 elements a group, padded to 96
    o2 = pk.add(None, count=24)
    o3 = pk.interleave([c, d], 2)
    o4 = pk.add(a.to(BF16))                             # a parameter that is not fp32
    buf = pk.build(a.device)
    assert torch.equal(buf[o1:o2].view(3, 96), TF.pad((a * 0.5).to(BF16).view(3, 80), (0, 16)))
    assert not buf[o2:o3].any()
    assert torch.equal(buf[o3:o4].view(2, 2, 32), torch.stack([c.to(BF16).view(2, 32), d.to(BF16).view(2, 32)], 1))
    assert torch.equal(buf[o4:o4 + 240], a.to(BF16).view(-1))


@pytest.mark.parametrize("n", [8, 128, 200, 264])
@pytest.mark.parametrize("k", [64, 256, 264])
@pytest.mark.parametrize("dtype", [F32, BF16])
def test_batched_products_on_both_sides_of_the_epilogue_rule(n, k, dtype):
    """Four K blocks and fewer drain with eight warps; enough tiles that every CTA reuses its staging tiles."""
    from bioemu2_b200 import functional as F

    g = _gen(n, k)
    a, b = (torch.randn(300, r, k, generator=g).to(BF16).cuda() for r in (130, n))
    out = torch.empty(300, 130, n, dtype=dtype, device="cuda")
    _close(F.bmm_nt_into(a, b, out), torch.einsum("bik,bjk->bij", a.float(), b.float()))
