"""The float32 product on the tensor cores (csrc/float_gemm.cu) against float64, at the edges of its tiles, steps and splits."""

from pathlib import Path

import pytest
import torch

from dli_b200.csrc import build
from dli_b200.kernels import gemm, ops


def _error(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.gpu
@pytest.mark.parametrize("tile,splits", [(0, 0), (32, 1), (32, 8), (64, 1), (64, 2), (128, 1), (128, 4)])
@pytest.mark.parametrize("batch,tokens,features,K", [(0, 1, 1, 4), (0, 31, 127, 60), (3, 33, 129, 68), (0, 64, 128, 128), (2, 65, 8, 192), (0, 127, 257, 516), (0, 129, 100, 1028)])
def test_products_at_the_edges_of_tiles(batch, tokens, features, K, tile, splits):
    g = torch.Generator().manual_seed(tokens + K)
    x, w = ([torch.randn(*([batch] if batch else []), rows, K, generator=g).cuda() for rows in (tokens, features)])
    want = x.double() @ w.double().transpose(-1, -2)
    # exact products, sums of at most 8 truncated additions (2^-23 each, with one sign) and of K / 64 rounded ones: 5e-7 for these K
    assert _error(ops.float_gemm(x, w, tile=tile, splits=splits), want) <= 5e-7


@pytest.mark.gpu
def test_rows_of_a_wider_tensor_and_a_given_result():
    g = torch.Generator().manual_seed(1)
    x, w = torch.randn(40, 300, generator=g).cuda()[:, 4:264], torch.randn(90, 520, generator=g).cuda()[:, 260:]
    room = torch.full((40, 95), 7.0).cuda()
    ops.float_gemm(x, w, room[:, 3:93])
    assert _error(room[:, 3:93], x.double() @ w.double().t()) <= 5e-7 and (room[:, :3] == 7).all() and (room[:, 93:] == 7).all()
    with pytest.raises(ops.KernelError):
        ops.float_gemm(x[:, 1:], w[:, 1:])  # rows off their 16-byte boundaries
    assert _error(gemm.linear(x[:, 1:], w[:, 1:]), x[:, 1:].double() @ w[:, 1:].double().t()) <= 2e-6  # the library takes them


@pytest.mark.gpu
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.4e38])
@pytest.mark.parametrize("tile,splits", [(32, 1), (64, 4), (128, 1)])
def test_numbers_that_are_not_finite_stay_in_their_row_and_column(value, tile, splits):
    g = torch.Generator().manual_seed(2)
    x, w = torch.randn(70, 320, generator=g).cuda(), torch.randn(140, 320, generator=g).cuda() * 0.1
    x[5, 7], w[133, 300] = value, value
    got, want = ops.float_gemm(x, w, tile=tile, splits=splits), (x.double() @ w.double().t()).float()
    rest = torch.ones(70, 140, dtype=torch.bool)
    rest[5], rest[:, 133] = False, False
    assert _error(got[rest], want.double()[rest]) <= 5e-7
    assert (got.isnan() == want.isnan()).all() and (got.isinf() == want.isinf()).all() and (got[want.isinf()] == want[want.isinf()]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("x_power,w_power", [(-118, 0), (-126, 0), (0, -126), (-140, 60), (60, -140), (-70, -50), (90, -90), (110, -60), (40, 60)])
@pytest.mark.parametrize("splits", [1, 4])
def test_numbers_of_any_size(x_power, w_power, splits):
    """The third term of a float32 number, 2^-17 and less of it, counts down to the smallest numbers; what is too large for the terms is computed again."""
    g = torch.Generator().manual_seed(4)
    x, w = (torch.randn(40, 320, generator=g).double() * 2.0**x_power).float().cuda(), (torch.randn(130, 320, generator=g).double() * 2.0**w_power).float().cuda()
    # as above 5e-7; computed again by 320 additions one after another, of which the sum's last bits see some sqrt(320) 2^-24, 1.1e-6, twice that for scatter
    assert _error(ops.float_gemm(x, w, tile=32, splits=splits), x.double() @ w.double().t()) <= (2.2e-6 if x_power > 100 or x_power + w_power > 75 else 5e-7)


@pytest.mark.gpu
@pytest.mark.parametrize("x_power,w_power", [(-110, 0), (0, -110), (-118, 0), (60, -118), (-126, 40), (-60, -60), (90, -90), (40, 60)])
@pytest.mark.parametrize("splits", [1, 4])
def test_numbers_of_any_size(x_power, w_power, splits):
    """The three terms are the number down to 2^-110, from there on but for 2^-134."""
    g = torch.Generator().manual_seed(4)
    x, w = (torch.randn(40, 320, generator=g).double() * 2.0**x_power).float().cuda(), (torch.randn(130, 320, generator=g).double() * 2.0**w_power).float().cuda()
    # as above 5e-7; beside it up to 2^-134 of numbers around 2^power
    assert _error(ops.float_gemm(x, w, tile=32, splits=splits), x.double() @ w.double().t()) <= 5e-7 + 2.0 ** (-134 - min(x_power, w_power))


@pytest.mark.gpu
@pytest.mark.parametrize("tile,splits,skip", [(32, 2, 7), (64, 4, 0), (128, 2, 3), (32, 1, 7)])
def test_a_wait_that_runs_out(tile, splits, skip):
    """One CTA of each cluster waits for terms that are never handed in: none of the cluster's CTAs stores what it would add up."""
    g = torch.Generator().manual_seed(skip)
    x, w = torch.randn(40, 512, generator=g).cuda(), torch.randn(140, 512, generator=g).cuda()
    assert ops.device_wait_errors() == {}
    out = torch.full((40, 140), 7.0, device="cuda")
    ops.float_gemm_wait_test(out, x, w, tile, splits, wait_limit=4000, skip_step=skip)
    torch.cuda.synchronize()  # returns: the kernel ended by itself
    assert (out == 7).all()
    assert ops.device_wait_errors()["float_gemm.cu"] in (1, 2, 3, 4) and ops.device_wait_errors() == {}
    assert _error(ops.float_gemm(x, w, tile=tile, splits=splits), x.double() @ w.double().t()) <= 5e-7
    assert ops.device_wait_errors() == {}


@pytest.mark.parametrize("tokens,features,K,own", [
    (8, 512, 256, False), (8, 1024, 256, True), (16, 512, 384, False), (8, 512, 512, True), (12, 320, 768, False), (16, 384, 768, True), (8, 64, 1024, True), (16, 64, 2048, True),
    (8, 64, 8192, False), (16, 256, 8192, False), (8, 320, 8192, True), (8, 32768, 2048, True), (8, 32768, 4096, False), (12, 32768, 4096, True), (8, 8192, 2048, True),
    (8, 16384, 8192, True), (16, 32, 4096, True), (16, 32, 8192, False)])
def test_which_products_of_few_tokens_go_there(tokens, features, K, own):
    """Small products and few features with long sums stay with the library up to 16 tokens."""
    assert gemm._float_few(tokens, features, K) == own


def test_more_tiles_than_a_grid_has_stay_with_the_library():
    x, w = torch.empty(256), torch.empty(8, 256)
    assert ops.float_gemm_supported(x.expand(65535 * 128, 256), w) and not ops.float_gemm_supported(x.expand(65535 * 128 + 1, 256), w)
    assert ops.float_gemm_supported(x.expand(65535, 8, 256), w.expand(65535, 8, 256)) and not ops.float_gemm_supported(x.expand(65536, 8, 256), w.expand(65536, 8, 256))
    assert not ops.float_gemm_supported(x.expand(8, 256), w.to("meta"))


@pytest.mark.gpu
def test_as_many_products_as_a_grid_has():
    x, w = torch.ones(1, 1, 256, device="cuda").expand(65535, 33, 256), torch.full((1, 1, 256), 0.5, device="cuda").expand(65535, 3, 256)
    out = ops.float_gemm(x, w)  # in tiles of 32 there would be twice as many
    assert out.shape == (65535, 33, 3) and (out == 128).all()


def test_no_kernel_loads_by_the_non_coherent_path():
    """Kernels start while the one in front still runs (programmatic launches), and its end orders ordinary loads only."""
    sources = sorted(p for p in Path(build.__file__).parent.iterdir() if p.suffix in (".cu", ".cuh", ".h"))
    assert len(sources) > 20
    assert [p.name for p in sources if "ld.global.nc" in p.read_text() or "__ldg(" in p.read_text()] == []
