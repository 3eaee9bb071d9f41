"""The gated norm over parts of a row, several parts to a warp (csrc/ssm.cu: gated_part_rmsnorm_kernel), at the sizes where its lanes and runs change, with
counts that leave the last warp partly empty."""

import pytest
import torch

from dli_b200.kernels import ops
from tests import cpu_ops as ref


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-6), (torch.bfloat16, 5e-3)])  # a few float32 roundings; one rounding to bfloat16 (2^-9) at full size
@pytest.mark.parametrize("n,parts", [(1, 1), (3, 5), (33, 2), (683, 3)])  # (from 2,048 parts on other kernels take parts of 257 to 512)
@pytest.mark.parametrize("size", [8, 32, 40, 64, 72, 128, 136, 256, 264, 512, 520, 1024, 1032])
def test_parts(size, n, parts, dtype, tol):
    g = torch.Generator().manual_seed(size + n)
    inner = size * parts
    y, u = torch.randn(n, inner, generator=g) * 2, torch.randn(n, inner + 16, generator=g).to(dtype)
    w, div = 1 + 0.1 * torch.randn(inner, generator=g), torch.rand(n, parts, generator=g) + 0.5
    for more in ({}, {"gate_after": True}, {"gate_after": True, "gate": "sigmoid", "divisor": div}):
        want, got = torch.empty(n, inner, dtype=dtype), torch.full((n, inner), float("nan"), dtype=dtype, device="cuda")
        ref.gated_group_rmsnorm(want, y, u, 8, w, parts, 1e-6, **more)
        on_gpu = {k: v.cuda() if isinstance(v, torch.Tensor) else v for k, v in more.items()}
        ops.gated_group_rmsnorm(got, y.cuda(), u.cuda(), 8, w.cuda(), parts, 1e-6, **on_gpu)
        err = (got.cpu().float() - want.float()).abs().max()
        assert err <= tol * max(1.0, want.float().abs().max()), (more, float(err))


@pytest.mark.gpu
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("size,n", [(24, 3), (72, 3), (264, 3), (264, 683), (520, 3)])
def test_a_gate_that_is_not_finite_counts_once(size, n, value):
    """Lanes without numbers of their own add nothing to the part's sum, whatever stands in the part's last numbers."""
    parts, g = 3, torch.Generator().manual_seed(size)
    y, u, w = torch.randn(n, size * parts, generator=g), torch.randn(n, size * parts, generator=g), torch.ones(size * parts)
    u[1, size - 1] = value
    for more in ({}, {"gate_after": True}):
        want, got = torch.empty(n, size * parts), torch.zeros(n, size * parts, device="cuda")
        ref.gated_group_rmsnorm(want, y, u, 0, w, parts, 1e-6, **more)
        ops.gated_group_rmsnorm(got, y.cuda(), u.cuda(), 0, w.cuda(), parts, 1e-6, **more)
        fine, got = want.isfinite(), got.cpu()
        assert (got.isnan() == want.isnan()).all() and (got.isinf() == want.isinf()).all() and (got[fine] - want[fine]).abs().max() <= 1e-5
