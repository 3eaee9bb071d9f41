"""The product of some tokens (csrc/few_gemm.cu) against float64, at the edges of its tiles, steps and splits, and which products it serves."""

import pytest
import torch

from dli_b200.kernels import gemm, ops


def _error(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.gpu
@pytest.mark.parametrize("splits", [1, 2, 4, 8])
@pytest.mark.parametrize("tokens,features,K", [(1, 4, 8), (9, 132, 120), (16, 128, 128), (17, 300, 136), (33, 128, 1032), (64, 260, 2048), (65, 124, 384), (127, 256, 256), (128, 12, 1024)])
def test_products_at_the_edges_of_tiles(tokens, features, K, splits):
    g = torch.Generator().manual_seed(tokens + K)
    room, w = torch.randn(tokens, K + 24, generator=g).bfloat16().cuda(), torch.randn(features, K, generator=g).bfloat16().cuda()
    x = room[:, 8 : 8 + K]  # rows of a wider tensor
    got = ops.few_gemm(x, w, splits)
    # one rounding to bfloat16, 2^-9 at most and 2^-9 / sqrt(3) in the mean; float32 sums add 1e-6
    assert got.shape == (tokens, features) and _error(got, x.double() @ w.double().t()) <= 2.0**-9


@pytest.mark.gpu
@pytest.mark.parametrize("splits", [1, 2, 4])
@pytest.mark.parametrize("tokens,I,K", [(9, 64, 128), (50, 192, 520), (96, 128, 1024)])
def test_the_activation_of_a_gated_feed_forward(tokens, I, K, splits):
    g = torch.Generator().manual_seed(tokens)
    x, gate, up = torch.randn(tokens, K, generator=g).bfloat16().cuda(), (torch.randn(I, K, generator=g) * 0.1).bfloat16().cuda(), (torch.randn(I, K, generator=g) * 0.1).bfloat16().cuda()
    w = torch.stack([gate.view(-1, 64, K), up.view(-1, 64, K)], 1).reshape(2 * I, K).contiguous()
    a, b = (x.double() @ gate.double().t()).bfloat16(), (x.double() @ up.double().t()).bfloat16()  # the sums as bfloat16 holds them
    want = torch.nn.functional.silu(a.double()) * b.double()
    # a sum near the middle between two bfloat16 numbers may be rounded the other way: some of them move by 2^-8, on top of the result's own 2^-9
    assert _error(ops.few_gemm(x, w, splits, swiglu=True), want) <= 2.0**-8


@pytest.mark.gpu
@pytest.mark.parametrize("splits,skip", [(1, 2), (2, 5), (2, 0), (4, 7)])
def test_a_wait_that_runs_out(splits, skip):
    """One CTA of each cluster misses a step's copies: none of the cluster's CTAs stores what it would add up, the code is read once, the next product is right."""
    g = torch.Generator().manual_seed(skip)
    K = 512 if splits == 1 else 1024
    x, w = torch.randn(17, K, generator=g).bfloat16().cuda(), torch.randn(300, K, generator=g).bfloat16().cuda()
    assert ops.device_wait_errors() == {}
    out = torch.full((17, 300), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.few_gemm_wait_test(out, x, w, splits, wait_limit=4000, skip_step=skip)
    torch.cuda.synchronize()  # returns: the kernel ended by itself
    assert (out == 7).all()
    assert ops.device_wait_errors()["few_gemm.cu"] in (2, 3) and ops.device_wait_errors() == {}
    assert _error(ops.few_gemm(x, w, splits), x.double() @ w.double().t()) <= 2.0**-9
    assert ops.device_wait_errors() == {}


def test_which_products_go_there():
    def takes(tokens, features, K, dtype=torch.bfloat16, swiglu=False):
        return gemm.few_product(torch.empty(tokens, K, dtype=dtype), torch.empty(features, K, dtype=dtype), swiglu)

    assert takes(24, 2048, 2048) and not takes(25, 2048, 2048) and takes(64, 2048, 8192) and not takes(65, 2048, 8192) and not takes(8, 2048, 2048)
    assert takes(24, 10304, 2048) and not takes(25, 10304, 2048) and not takes(16, 2048, 512) and not takes(16, 64, 2048)
    assert takes(96, 16384, 2048, swiglu=True) and not takes(97, 16384, 2048, swiglu=True) and not takes(16, 2048, 2048, torch.float32)
    assert not gemm.few_product(torch.empty(16, 2052, dtype=torch.bfloat16)[:, 4:], torch.empty(2048, 2048, dtype=torch.bfloat16))  # rows off 16 bytes
    assert [gemm.few_splits(*s) for s in ((2048, 2048), (16384, 2048), (1024, 4096), (4240, 2048), (4096, 4096), (1024, 1024))] == [4, 1, 8, 2, 4, 2]


@pytest.mark.parametrize("features,K,swiglu,most", [
    (18944, 2048, False, 24), (19072, 2048, False, 0), (20608, 4096, False, 0), (28672, 2048, False, 24), (28672, 1024, False, 0), (38016, 2048, False, 0), (37888, 4096, False, 24),
    (19200, 4096, True, 0), (28672, 4096, True, 64), (28672, 1024, True, 24), (57344, 4096, True, 24), (11264, 8192, True, 64), (18944, 8192, True, 96), (16384, 2048, True, 96),
    (4096, 4096, False, 40), (2048, 4096, False, 64), (4096, 8192, False, 64), (1024, 4096, False, 64), (6144, 4096, False, 16), (12352, 4096, False, 24),
    (5376, 2048, False, 16), (6176, 2048, False, 12), (8192, 2048, False, 0), (10304, 2048, False, 24), (4096, 2048, False, 24), (4096, 1024, False, 24), (1024, 1024, False, 16)])
def test_up_to_how_many_tokens(features, K, swiglu, most, monkeypatch):
    """The lines lie where both sides were measured: a second wave of tiles, CTAs that share K in pairs, and wide products of some more tokens cost more than the library's."""
    monkeypatch.setattr(gemm, "sm_count", lambda: 148)
    assert gemm.few_max_tokens(features, K, swiglu) == most


def test_rows_that_do_not_lie_behind_one_another_stay_with_the_library():
    w = torch.empty(2048, 2048, dtype=torch.bfloat16)
    assert gemm.few_product(torch.empty(16, 2056, dtype=torch.bfloat16)[:, :2048], w) and not gemm.few_product(torch.empty(1, 2048, dtype=torch.bfloat16).expand(16, -1), w)
    assert not gemm.few_product(torch.empty(4096, dtype=torch.bfloat16).as_strided((16, 2048), (8, 1)), w)
    assert not ops.few_gemm_supported(torch.empty(16, 2048, dtype=torch.bfloat16), torch.empty(2048, 2048, dtype=torch.bfloat16, device="meta"))  # on another device


@pytest.mark.gpu
def test_an_expanded_row():
    g = torch.Generator().manual_seed(3)
    x, w = torch.randn(1, 2048, generator=g).bfloat16().cuda().expand(16, -1), torch.randn(1024, 2048, generator=g).bfloat16().cuda()
    assert _error(gemm.linear(x, w), x.double() @ w.double().t()) <= 2.0**-9
