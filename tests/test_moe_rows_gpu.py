"""Rows to the experts and their outputs back (csrc/moe_sort.cu: moe_gather_kernel, csrc/moe_combine.cu) at the edges of a warp's pieces and of the choices that are
looked up together."""

import pytest
import torch

from dli_b200.kernels import ops
from tests import cpu_ops as ref


@pytest.mark.gpu
@pytest.mark.parametrize("W,E,identity,top", [(1032, 6, 0, 4), (2056, 5, 3, 7), (1024, 40, 4, 35), (264, 7, 6, 8)])
@pytest.mark.parametrize("n", [9, 300])  # sorted in one launch, and in several (from 2,049 pairs on)
def test_rows_there_and_back(W, E, identity, top, n):
    g = torch.Generator().manual_seed(W)
    x = torch.randn(n, W, generator=g).bfloat16()
    w_up, w_down = ((torch.randn(E, *s, generator=g) * s[1] ** -0.5).bfloat16() for s in ((64, W), (W, 64)))
    ids = torch.stack([torch.randperm(E + identity, generator=g)[:top] for _ in range(n)]).int()
    weights = torch.rand(n, top, generator=g)
    want, got = torch.zeros(n, W), torch.full((n, W), 7.0, dtype=torch.bfloat16, device="cuda")
    ref.moe_experts(want, x.float(), ids, weights, w_up.float(), w_down.float(), "relu2", gated=False)
    ops.moe_combine(got, ops.moe_products(x.cuda(), ids.cuda(), weights.cuda(), w_up.cuda(), w_down.cuda(), "relu2", gated=False, few=False))
    # hidden rows and the result are rounded to bfloat16 (2^-9 each), sums are float32
    assert (got.float().cpu() - want).norm() <= 5e-3 * want.norm()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("E,groups,W,n", [(6, 1, 264, 257), (753, 1, 256, 261), (1504, 32, 8, 258), (1520, 1, 264, 257), (5, 1, 2056, 1185), (9, 3, 264, 2368), (9, 3, 264, 2371)])
def test_routing_of_many_tokens(E, groups, W, n, dtype):
    """In either form of the kernel, and with more experts than fit a block of four tokens, a token's experts and weights are those of the kernel for few tokens, to the last
    bit: every sum has the same order."""
    g = torch.Generator().manual_seed(E)
    x, router, corr = torch.randn(n, W, generator=g).to(dtype).cuda(), (torch.randn(E, W, generator=g) * 0.1).cuda(), torch.randn(E, generator=g).cuda() * 0.1
    ids, weights = torch.empty(n, 3, dtype=torch.int32, device="cuda"), torch.empty(n, 3, device="cuda")
    few = torch.empty_like(ids), torch.empty_like(weights)
    ops.moe_route(ids, weights, x, router, corr, groups, max(1, groups // 2), 1.5)
    for first in range(0, n, 200):
        ops.moe_route(few[0][first : first + 200], few[1][first : first + 200], x[first : first + 200], router, corr, groups, max(1, groups // 2), 1.5)
    assert torch.equal(ids, few[0]) and torch.equal(weights, few[1])
