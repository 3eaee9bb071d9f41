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
