"""The matrix memory in tiles of 128 tokens (csrc/matrix_memory_umma.cu) against the recurrence in float64, at the edges of its tiles, segments and column blocks."""

import pytest
import torch

from dli_b200.kernels import ops
from tests.test_ssm_tiles_gpu import _same_kind

CAP = 15.0


def _inputs(H, d, dv, lens, seed, rows=0):
    g = torch.Generator().manual_seed(seed)
    n, S = sum(lens) + rows, len(lens)
    u, gates = torch.randn(n, H * (2 * d + dv) + 8, generator=g).bfloat16(), torch.randn(n, 2 * H, generator=g)
    bias = torch.cat([torch.rand(H, generator=g) * 10 - 10, torch.rand(H, generator=g) * 3 + 3])
    top = torch.randn(S, H, 1, generator=g).expand(S, H, dv + 1).contiguous()
    return u, gates, bias, torch.randn(S, H, dv + 1, d, generator=g), top


def _exact(u, gates, bias, state, top, lens):
    _, H, dv1, d = state.shape
    u, gates, bias, state, top = u.double(), gates.double(), bias.double(), state.double(), top.double().clone()
    o, div, t0 = [], [], 0
    for s, n in enumerate(lens):
        S, m = state[s], top[s, :, 0]
        for t in range(t0, t0 + n):
            q, k = u[t, : H * d].view(H, d) * d**-0.5, u[t, H * d : 2 * H * d].view(H, d)
            v = torch.cat([u[t, 2 * H * d : 2 * H * d + H * (dv1 - 1)].view(H, dv1 - 1), torch.ones(H, 1, dtype=torch.float64)], 1)
            i, f = CAP * torch.tanh((gates[t, :H] + bias[:H]) / CAP), torch.nn.functional.logsigmoid(CAP * torch.tanh((gates[t, H:] + bias[H:]) / CAP))
            new = torch.fmax(f + m, i)  # (a NaN does not become the maximum)
            S = torch.exp(f + m - new)[:, None, None] * S + torch.exp(i - new)[:, None, None] * v[:, :, None] * k[:, None, :]
            m = new
            read = (S @ q[:, :, None])[..., 0]
            o.append(read[:, :-1].reshape(-1)), div.append(torch.fmax(read[:, -1].abs(), torch.exp(-m)) + 1e-6)
        state[s], top[s] = S, m[:, None]
        t0 += n
    return torch.stack(o), torch.stack(div), state, top


def _run(inputs, lens, order, **how):
    u, gates, bias, state, top = [x.cuda() for x in inputs]
    S, H, dv1, d = state.shape
    o, div = torch.full((u.shape[0], H * (dv1 - 1)), 7.0).cuda(), torch.full((u.shape[0], H), 7.0).cuda()
    state, top = state[order].contiguous(), top[order].contiguous()
    slots = torch.empty(S, dtype=torch.int32)
    slots[order] = torch.arange(S, dtype=torch.int32)
    q_start = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32).cuda()
    ops.matrix_memory_scan(o, div, u, gates, bias, CAP, state, top, q_start, slots.cuda(), max_len=max(lens), **how)
    back = torch.empty_like(state), torch.empty_like(top)
    back[0][order], back[1][order] = state, top
    return [x.cpu() for x in (o, div, *back)]


@pytest.mark.gpu
@pytest.mark.parametrize("H,d,dv,lens", [(9, 128, 128, [1, 4, 5, 127]), (2, 48, 72, [128, 129, 49]), (1, 112, 8, [257, 3]), (3, 32, 136, [513]), (2, 64, 64, [1, 700])])
def test_tiles_of_128_tokens(H, d, dv, lens):
    inputs = _inputs(H, d, dv, lens, d + dv, rows=5)
    inputs[0][sum(lens) :] = float("nan")  # rows behind the last token belong to no sequence
    want = _exact(inputs[0], inputs[1], inputs[2], inputs[3].clone(), inputs[4], lens)
    order, n, walked = torch.arange(len(lens) - 1, -1, -1), sum(lens), None
    for how in ({"form": "walk"}, *({"form": "chunk", "segments": s, "tile": 128} for s in (0, 1, 3, 9))):
        o, div, state, top = _run(inputs, lens, order, **how)
        errors = [float((a.double() - b).norm() / b.norm()) for a, b in ((o[:n], want[0]), (div[:n], want[1]), (state, want[2]), (top, want[3]))]
        walked = walked or errors
        # float32: six roundings of 2^-24 a token that add up at random over at most 700 tokens, 9.5e-6 with twice that for scatter; tiles no worse than the walk
        assert all(e <= min(1.9e-5, max(1e-6, 2 * w)) for e, w in zip(errors, walked)), (how, errors, walked)
        assert (o[n:] == 7.0).all() and (div[n:] == 7.0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("where", ["q", "k", "v", "gate", "state"])
@pytest.mark.parametrize("bad", [0, 127, 128, 299, 310])
def test_infinities_and_nans_stay_where_the_recurrence_has_them(where, value, bad):
    """A number that is not finite reaches its own and later tokens of its own sequence, and no other (token 310 is the next sequence's)."""
    H, d, dv, lens = 2, 48, 72, [300, 20]
    inputs = _inputs(H, d, dv, lens, 11)
    u, gates, _, state, _ = inputs
    if where == "state":
        state[0, 1, bad % dv, 3] = value
    elif where == "gate":
        gates[bad, 1 + bad % 2 * 2] = value
    else:
        u[bad, {"q": d, "k": (H + 1) * d, "v": 2 * H * d + dv}[where] + 3] = value
    want = _exact(inputs[0], inputs[1], inputs[2], state.clone(), inputs[4], lens)
    for segments in (1, 3):
        for a, b in zip(_run(inputs, lens, torch.arange(2), form="chunk", segments=segments, tile=128), want):
            assert _same_kind(a, b, 4e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("skip", [0, 1])
def test_a_wait_that_runs_out(skip):
    """The copies of q and k of one tile never come: no read-outs or divisors of that tile or a later one, no states and no maxima are stored, the next step is right."""
    H, d, dv, lens = 2, 48, 72, [300, 290]
    inputs = _inputs(H, d, dv, lens, 5)
    want = _exact(inputs[0], inputs[1], inputs[2], inputs[3].clone(), inputs[4], lens)
    q_start, slot = torch.tensor([0, 300, 590], dtype=torch.int32).cuda(), torch.arange(2, dtype=torch.int32).cuda()
    assert ops.device_wait_errors() == {}
    u, gates, bias, state, top = [x.cuda() for x in inputs]
    o, div = torch.full((590, H * dv), 7.0).cuda(), torch.full((590, H), 7.0).cuda()
    ops.matrix_memory_umma_wait_test(o, div, u, gates, bias, CAP, state, top, q_start, slot, wait_limit=20000, skip_tile=skip)
    torch.cuda.synchronize()  # returns: the kernel ended by itself
    assert torch.equal(state.cpu(), inputs[3]) and torch.equal(top.cpu(), inputs[4])
    for first, last in ((0, 300), (300, 590)):
        for got, exact in ((o, want[0]), (div, want[1])):
            assert _same_kind(got[first : first + 128 * skip].cpu(), exact[first : first + 128 * skip], 4e-6) and (got[first + 128 * skip : last] == 7).all()
    assert "matrix_memory_umma.cu" in ops.device_wait_errors() and ops.device_wait_errors() == {}
    for a, b in zip(_run(inputs, lens, torch.arange(2), form="chunk", segments=1, tile=128), want):
        assert _same_kind(a, b, 4e-6)
    assert ops.device_wait_errors() == {}
