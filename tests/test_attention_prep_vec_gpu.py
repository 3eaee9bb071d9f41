"""What lies between an attention's projections and its kernel, in pieces of 16 bytes (csrc/diff_attention.cu: diff_prep_vec_kernel, csrc/attention_prep.cu:
latent_prep_vec_kernel), against the kernels for any column and stride, which rows of an odd number of columns take, and against 64 bits."""

import pytest
import torch

from dli_b200.kernels import ops


def _close(a, b):
    # the same float32 arithmetic but for the order of a sum of squares (some 2^-22 of it): after rounding to bfloat16 one step, 2^-7 of the number, at most
    assert ((a.float() - b.float()).abs() <= 2.0**-7 * b.float().abs() + 1e-6).all()


def _near(got, want):
    # one rounding to bfloat16 (seven bits behind the first), 2^-8 of the number at most; in front of it float32 sums, roots and products of numbers of up to some 10, each
    # 2^-24 of them: 2e-5, which may also move a rounding
    assert ((got.double().cpu() - want).abs() <= 2.0**-8 * want.abs() + 2e-5).all()


def _turns(pos, freq, amp):
    angle = (pos.float()[:, None] * freq.float()[None]).double()  # (the kernels' angle is the float32 product)
    return angle.cos() * amp, angle.sin() * amp


@pytest.mark.gpu
@pytest.mark.parametrize("dim,nh,nkv,vdim,rot", [(32, 3, 1, 8, 32), (64, 16, 4, 128, 64), (64, 40, 8, 128, 22), (128, 16, 4, 64, 0), (256, 20, 5, 256, 256)])
@pytest.mark.parametrize("writes", [True, False])
def test_differential(dim, nh, nkv, vdim, rot, writes):
    n, page, pages = 19, 8, 4
    g = torch.Generator().manual_seed(dim + nh)
    k_col, v_col = nh * 2 * dim, (nh + nkv) * 2 * dim
    wide = torch.randn(n, v_col + nkv * vdim + 1, generator=g).bfloat16().cuda()
    wq, wk, freq = ((torch.rand(k, generator=g) + 0.5).cuda() for k in (dim, dim, max(rot // 2, 1)))
    pos = torch.randint(0, 5000, (n,), generator=g, dtype=torch.int32).cuda()
    slots = torch.randperm(pages * page, generator=g)[:n].int().cuda()
    outs = []
    for proj in (wide[:, :-1].contiguous(), wide):
        q = torch.zeros(n, nh * 2 * dim, dtype=torch.bfloat16, device="cuda")
        k, v = (torch.zeros(pages, nkv, page, c, dtype=torch.bfloat16, device="cuda") for c in (2 * dim, vdim))
        ops.diff_prep(q, proj, k_col if writes else -1, v_col if writes else -1, wq, wk if writes else None, 1e-5, pos, freq, 1.25, slots if writes else None,
                      k if writes else None, v if writes else None, nh, nkv, dim, vdim, rot, page)
        outs.append((q, k, v))
    _close(outs[0][0], outs[1][0]), _close(outs[0][1], outs[1][1])
    assert torch.equal(outs[0][2], outs[1][2])
    x, cos, sin = wide[:, :-1].double().cpu(), *_turns(pos.cpu(), freq.cpu(), 1.25)
    for first, heads, weight, got in ((0, nh, wq, outs[0][0].view(n, nh, 2, dim)), (k_col, nkv, wk, outs[0][1].transpose(1, 2).reshape(pages * page, nkv, 2, dim)[slots.long()])):
        y = x[:, first : first + heads * 2 * dim].view(n, heads, 2, dim)
        y = y / (y.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * weight.double().cpu()
        a, b = y[..., 0:rot:2].clone(), y[..., 1:rot:2].clone()
        c, d = (z[:, None, None, : rot // 2] for z in (cos, sin))
        y[..., 0:rot:2], y[..., 1:rot:2] = a * c - b * d, b * c + a * d
        _near(got, y if first == 0 or writes else torch.zeros_like(y))


@pytest.mark.gpu
@pytest.mark.parametrize("nh,d,dr,r", [(1, 8, 16, 8), (16, 128, 64, 192), (130, 32, 64, 256), (64, 8, 128, 264), (5, 16, 48, 512)])
@pytest.mark.parametrize("writes", [True, False])
def test_latent(nh, d, dr, r, writes):
    n, page, pages = 19, 8, 4
    g = torch.Generator().manual_seed(nh)
    wide = torch.randn(n, nh * (d + dr) + r + dr + 1, generator=g).bfloat16().cuda()
    w, inv = ((torch.rand(k, generator=g) + 0.5).cuda() for k in (r, dr // 2))
    pos = torch.randint(0, 5000, (n,), generator=g, dtype=torch.int32).cuda()
    slots = torch.randperm(pages * page, generator=g)[:n].int().cuda()
    outs = []
    for columns in (wide.shape[1] - 1, wide.shape[1]):
        q, k = torch.zeros(n, nh * (r + dr), dtype=torch.bfloat16, device="cuda"), torch.zeros(pages, 1, page, r + dr, dtype=torch.bfloat16, device="cuda")
        ops.latent_prep(q, wide[:, :columns].contiguous(), w, 1e-5, pos, inv, slots if writes else None, k if writes else None, nh, d, dr, r, dr, page, 1.25)
        outs.append((q, k))
    _close(outs[0][0], outs[1][0]), _close(outs[0][1], outs[1][1])
    x, cos, sin = wide[:, :-1].double().cpu(), *_turns(pos.cpu(), inv.cpu(), 1.25)
    down = x[:, nh * (d + dr) :]

    def turned(part, c, s):
        lo, hi = part[..., : dr // 2], part[..., dr // 2 :]
        return torch.cat([lo * c - hi * s, hi * c + lo * s], -1)

    _near(outs[0][0].view(n, nh, r + dr)[..., r:], turned(x[:, : nh * (d + dr)].view(n, nh, d + dr)[..., d:], cos[:, None], sin[:, None]))
    if writes:
        latent = down[:, :r] / (down[:, :r].pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * w.double().cpu()
        _near(outs[0][1].view(pages * page, r + dr)[slots.long()], torch.cat([latent, turned(down[:, r:], cos, sin)], -1))
