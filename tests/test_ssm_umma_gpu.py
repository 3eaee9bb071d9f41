"""The selective scan in tiles of 128 tokens (csrc/ssm_umma.cu) at the edges of its tiles, segments and column blocks."""

import pytest
import torch

from dli_b200.kernels import ops
from tests.test_ssm_tiles_gpu import _exact, _same_kind


@pytest.mark.gpu
@pytest.mark.parametrize("dt_shift", [-5.0, 40.0], ids=["long_memory", "no_memory"])
@pytest.mark.parametrize("H,P,N,groups,lens", [(9, 64, 128, 3, [1, 4, 5, 127]), (4, 72, 48, 2, [128, 129, 31, 33]), (2, 136, 112, 1, [257, 3]), (3, 8, 32, 1, [700]), (2, 96, 64, 2, [1, 513])])
def test_tiles_of_128_tokens(H, P, N, groups, lens, dt_shift):
    g = torch.Generator().manual_seed(P + N)
    n, S = sum(lens), len(lens)
    xbc, u = torch.randn(n + 5, H * P + 2 * groups * N, generator=g).bfloat16(), torch.randn(n + 5, H + 1, generator=g).bfloat16()
    xbc[n:] = float("nan")  # rows behind the last token belong to no sequence
    vec = [torch.randn(H, generator=g) + dt_shift, torch.rand(H, generator=g) * 2.5, torch.randn(H, generator=g)]
    state = torch.randn(S, H, P, N, generator=g)
    want = _exact(xbc, u, 1, *vec, state.clone(), lens, groups)
    q_start, slot = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device="cuda"), torch.arange(S - 1, -1, -1, dtype=torch.int32, device="cuda")
    errors = {}
    for form, segments in (("walk", 0), ("chunk", 0), ("chunk", 1), ("chunk", 3), ("chunk", 9)):
        y, st = torch.full((n + 5, H * P), 7.0, device="cuda"), state.flip(0).cuda()
        ops.ssm_scan(y, xbc.cuda(), u.cuda(), 1, *[v.cuda() for v in vec], st, q_start, slot, groups, max_len=max(lens), form=form, segments=segments, tile=128)
        errors[form, segments] = [float((a.cpu().double() - b).norm() / b.norm()) for a, b in ((y[:n], want[0]), (st.flip(0), want[1]))]
        # float32: some four roundings of 2^-24 a token that add up at random over at most 700 tokens, 6.3e-6 with twice that for scatter; tiles no worse than the walk
        assert all(e <= min(6.3e-6, max(4e-7, 2 * w)) for e, w in zip(errors[form, segments], errors["walk", 0])), errors
        assert (y[n:] == 7.0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("where", ["x", "B", "C", "dt", "state"])
@pytest.mark.parametrize("bad", [0, 127, 128, 299, 310])
def test_infinities_and_nans_stay_where_the_recurrence_has_them(where, value, bad):
    """A number that is not finite reaches its own and later tokens of its own sequence and columns, and no other (token 310 is the next sequence's)."""
    H, P, N, lens = 2, 72, 48, [300, 20]
    n, g = sum(lens), torch.Generator().manual_seed(11)
    xbc, u, state = torch.randn(n, H * P + 2 * N, generator=g).bfloat16(), torch.randn(n, H, generator=g).bfloat16(), torch.randn(2, H, P, N, generator=g)
    if where == "state":
        state[0, 1, bad % P, 3] = value
    elif where == "dt":
        u[bad, 1] = value
    else:
        xbc[bad, {"x": P + bad % P, "B": H * P + 3, "C": H * P + N + 3}[where]] = value
    vec = torch.randn(3, H, generator=g)
    vec[0] -= 3.0  # small steps: no decay of the whole sequence underflows in float32
    want = _exact(xbc, u, 0, vec[0], vec[1] * 0.1, vec[2], state.clone(), lens, 1)
    q_start, slot, vec = torch.tensor([0, 300, 320], dtype=torch.int32).cuda(), torch.arange(2, dtype=torch.int32).cuda(), vec.cuda()
    for segments in (1, 3):
        y, st = torch.zeros(n, H * P).cuda(), state.cuda()
        ops.ssm_scan(y, xbc.cuda(), u.cuda(), 0, vec[0], vec[1] * 0.1, vec[2], st, q_start, slot, 1, max_len=300, form="chunk", segments=segments, tile=128)
        assert _same_kind(y, want[0], 1e-6) and _same_kind(st, want[1], 1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("skip", [0, 1])
def test_a_wait_that_runs_out(skip):
    """The copies of B and C of one tile never come: no read-outs of that tile or a later one and no states are stored, the code is read once, the next scan is right."""
    H, P, N, lens = 3, 72, 48, [300, 290]
    n, g = sum(lens), torch.Generator().manual_seed(5)
    xbc, u, state = torch.randn(n, H * P + 2 * N, generator=g).bfloat16(), torch.randn(n, H, generator=g).bfloat16(), torch.randn(2, H, P, N, generator=g)
    vec = torch.randn(3, H, generator=g)
    vec[0] -= 3.0
    want = _exact(xbc, u, 0, *vec, state.clone(), lens, 1)
    q_start, slot, vec = torch.tensor([0, 300, 590], dtype=torch.int32).cuda(), torch.arange(2, dtype=torch.int32).cuda(), vec.cuda()
    assert ops.device_wait_errors() == {}
    y, st = torch.full((n, H * P), 7.0).cuda(), state.cuda()
    ops.ssm_umma_wait_test(y, xbc.cuda(), u.cuda(), 0, *vec, st, q_start, slot, 1, wait_limit=20000, skip_tile=skip)
    torch.cuda.synchronize()  # returns: the kernel ended by itself
    assert torch.equal(st.cpu(), state)
    for first, last in ((0, 300), (300, 590)):
        assert _same_kind(y[first : first + 128 * skip], want[0][first : first + 128 * skip], 1e-6) and (y[first + 128 * skip : last] == 7).all()
    assert "ssm_umma.cu" in ops.device_wait_errors() and ops.device_wait_errors() == {}
    ops.ssm_scan(y, xbc.cuda(), u.cuda(), 0, *vec, st, q_start, slot, 1, max_len=300, form="chunk", segments=1, tile=128)
    assert _same_kind(y, want[0], 1e-6) and _same_kind(st, want[1], 1e-6) and ops.device_wait_errors() == {}
