"""The attention core at the edges of its two kernels: tile and row-block boundaries, an odd number of lines, and logits far
outside the range in which a row's softmax reference stays put; against a plain fp32 softmax."""
import pytest
import torch

from gpu_util import assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dh", [32, 48])
@pytest.mark.parametrize("N,lines,scale", [(1, 1, 1.0), (7, 3, 1.0), (127, 2, 1.0), (128, 3, 40.0), (129, 5, 1.0), (256, 3, 1.0),
                                           (257, 2, 40.0), (300, 3, 100.0), (512, 3, 1.0), (513, 2, 1.0)])
def test_attention_core_edges(N, lines, scale, dh):
    from bioemu2_b200 import _lib
    from bioemu2_b200 import functional as F

    g = torch.Generator().manual_seed(1000 + N)
    H = 2
    q, k, v = (torch.randn(lines, N, H, dh, generator=g).bfloat16() for _ in range(3))
    bias = scale * torch.randn(1, H, N, N, generator=g)
    if scale > 1:  # the maximum of a row grows from key tile to key tile
        bias += scale * torch.arange(N)[None, None, None, :] / 64
    mask = torch.rand(lines, N, generator=g) > 0.2
    mask[-1] = False                      # a line without a valid key averages over all keys
    bias_bf = (bias * F.LOG2E).bfloat16().float() / F.LOG2E   # the kernel takes the bias in bf16, base 2
    qs = (q.float() * (F.LOG2E / dh ** 0.5)).bfloat16().float() / F.LOG2E
    logits = torch.einsum("bqhd,bkhd->bhqk", qs, k.float()) + bias_bf
    logits = torch.where(mask[:, None, None, :], logits, torch.full_like(logits, -1e6))
    ref = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(logits.double(), -1), v.double())
    out = F.attention_core(q.cuda(), k.cuda(), v.cuda(), bias.cuda(), mask.cuda(), bias_div=lines)
    assert _lib.device_status() == 0
    assert_close(f"attention_core_N{N}_dh{dh}", out, ref)


@pytest.mark.parametrize("dh", [32, 48])
@pytest.mark.parametrize("rise_at", [None, 40, 64, 128, 200])
@pytest.mark.parametrize("masked", [False, True])
def test_rows_that_start_low(rise_at, masked, dh):
    """Live keys whose logits lie so far below zero that a row's reference moves down with the first half tile, and back up where
    later keys are more than the range above it: within the first half tile, from its second half, from the second tile.  Rows of
    one warp differ, so that only some of them move."""
    from bioemu2_b200 import _lib
    from bioemu2_b200 import functional as F

    g = torch.Generator().manual_seed(77)
    N, lines, H = 230, 3, 2
    q, k, v = (torch.randn(lines, N, H, dh, generator=g).bfloat16() for _ in range(3))
    bias = torch.randn(1, H, N, N, generator=g)
    bias[:, :, ::3] -= 90.0                # natural units: 130 in base 2
    bias[:, :, 1::6] += 50.0               # others leave the range upwards
    if rise_at is not None:
        bias[:, :, ::6, rise_at:] += 95.0
    mask = torch.ones(lines, N, dtype=torch.bool)
    if masked:
        mask = torch.rand(lines, N, generator=g) > 0.2
        mask[1, :64] = False               # the first half tile holds no valid key
    bias_bf = (bias * F.LOG2E).bfloat16().float() / F.LOG2E   # the kernel takes the bias in bf16, base 2
    qs = (q.float() * (F.LOG2E / dh ** 0.5)).bfloat16().float() / F.LOG2E
    logits = torch.einsum("bqhd,bkhd->bhqk", qs, k.float()) + bias_bf
    logits = torch.where(mask[:, None, None, :], logits, torch.full_like(logits, -1e6))
    ref = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(logits.double(), -1), v.double())
    out = F.attention_core(q.cuda(), k.cuda(), v.cuda(), bias.cuda(), mask.cuda(), bias_div=lines)
    assert _lib.device_status() == 0
    assert_close(f"attention_core_low_{rise_at}_{masked}_dh{dh}", out, ref)


@pytest.mark.parametrize("dh", [32, 48])
@pytest.mark.parametrize("N", [1, 63, 65, 128, 150, 192, 203, 256, 449, 512, 700])
@pytest.mark.parametrize("shift", [0.0, -90.0])
def test_half_tiles_without_a_valid_key(N, shift, dh):
    """Runs of masked keys that cover half tiles of 64 -- at the end, at the start, in the middle, everywhere -- with the rows'
    reference at 0 and away from it.  Bound: P and V in bf16, 2^-9 each, as in the tests above."""
    from bioemu2_b200 import _lib
    from bioemu2_b200 import functional as F

    g = torch.Generator().manual_seed(4000 + N)
    lines, H = 7, 2
    q, k, v = (torch.randn(lines, N, H, dh, generator=g).bfloat16() for _ in range(3))
    bias = torch.randn(1, H, N, N, generator=g)
    bias[:, :, ::3] += shift
    mask = torch.ones(lines, N, dtype=torch.bool)
    mask[0, N - N // 3:] = False            # padding
    mask[1, :N // 2] = False                # nothing but masked keys at first, then valid ones
    mask[2, N // 4:3 * N // 4] = False      # a hole
    mask[3] = False
    mask[4, 1:] = False                     # a single valid key
    mask[5, :-1] = False
    bias_bf = (bias * F.LOG2E).bfloat16().float() / F.LOG2E   # the kernel takes the bias in bf16, base 2
    qs = (q.float() * (F.LOG2E / dh ** 0.5)).bfloat16().float() / F.LOG2E
    logits = torch.einsum("bqhd,bkhd->bhqk", qs, k.float()) + bias_bf
    logits = torch.where(mask[:, None, None, :], logits, torch.full_like(logits, -1e6))
    ref = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(logits.double(), -1), v.double())
    out = F.attention_core(q.cuda(), k.cuda(), v.cuda(), bias.cuda(), mask.cuda(), bias_div=lines)
    assert _lib.device_status() == 0
    assert_close(f"attention_core_runs_{N}_{shift}_dh{dh}", out, ref)
