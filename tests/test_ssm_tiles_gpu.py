"""The selective scan over tiles of tokens (csrc/ssm_tc.cu) against the recurrence in float64, at the edges of its tiles, segments and column blocks."""

import pytest
import torch

from dli_b200.kernels import ops


def _exact(xbc, u, dt_col, dt_bias, a_log, d_skip, state, lens, groups):
    _, H, P, N = state.shape
    inner, out, t0 = H * P, [], 0
    state, xbc, u = state.double(), xbc.double(), u.double()
    for s, n in enumerate(lens):
        S = state[s]
        for t in range(t0, t0 + n):
            x = xbc[t, :inner].view(H, P)
            B = xbc[t, inner : inner + groups * N].view(groups, N).repeat_interleave(H // groups, 0)
            C = xbc[t, inner + groups * N :].view(groups, N).repeat_interleave(H // groups, 0)
            dt = torch.nn.functional.softplus(u[t, dt_col : dt_col + H] + dt_bias.double())
            S = torch.exp(-torch.exp(a_log.double()) * dt)[:, None, None] * S + (dt[:, None] * x)[:, :, None] * B[:, None, :]
            out.append(((S @ C[:, :, None])[..., 0] + d_skip.double()[:, None] * x).reshape(-1))
        state[s] = S
        t0 += n
    return torch.stack(out), state


@pytest.mark.gpu
@pytest.mark.parametrize("dt_shift", [-5.0, 0.0, 40.0], ids=["long_memory", "short_memory", "no_memory"])
@pytest.mark.parametrize("H,P,N,groups,lens", [
    (4, 64, 128, 2, [1, 64, 65, 200]), (2, 8, 8, 1, [16, 17, 63, 129]), (3, 72, 40, 3, [500]), (8, 64, 64, 1, [1, 1, 1, 33]), (2, 136, 16, 2, [128, 2]), (1, 64, 96, 1, [321])])
def test_tiles_and_segments(H, P, N, groups, lens, dt_shift):
    g = torch.Generator().manual_seed(len(lens) * 1000 + P + N)
    n, S, dt_col = sum(lens), len(lens), 3
    xbc = torch.randn(n, H * P + 2 * groups * N, generator=g).bfloat16()
    u = torch.randn(n, dt_col + H + 2, generator=g).bfloat16()
    dt_bias, a_log, d_skip = torch.randn(H, generator=g) + dt_shift, torch.rand(H, generator=g) * 2.5, torch.randn(H, generator=g)
    state = torch.randn(S, H, P, N, generator=g)
    y_ref, st_ref = _exact(xbc, u, dt_col, dt_bias, a_log, d_skip, state, lens, groups)
    q_start = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device="cuda")
    slot = torch.arange(S - 1, -1, -1, dtype=torch.int32, device="cuda")  # slots in another order than the sequences
    walked = None
    for form, segments in (("walk", 0), ("chunk", 0), ("chunk", 1), ("chunk", 2), ("chunk", 3), ("chunk", 7)):  # (seven: more than a sequence has tiles)
        y, st = torch.full((n, H * P), float("nan"), device="cuda"), state.flip(0).cuda()
        ops.ssm_scan(y, xbc.cuda(), u.cuda(), dt_col, dt_bias.cuda(), a_log.cuda(), d_skip.cuda(), st, q_start, slot, groups, max_len=max(lens), form=form, segments=segments, tile=64)
        errors = [float((a.cpu().double() - b).norm() / b.norm()) for a, b in ((y, y_ref), (st.flip(0), st_ref))]
        # float32: some four roundings of 2^-24 a token that add up at random over at most 500 tokens, 2.7e-6, and twice that for scatter
        assert all(e <= 5.4e-6 for e in errors), (form, segments, errors)
        if form == "walk":
            walked = errors
        else:  # no worse than the walk's by more than its scatter
            assert all(e <= max(2 * w, 4e-7) for e, w in zip(errors, walked)), (form, segments, errors, walked)


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["step size", "A_log"])
def test_a_gate_that_is_not_a_number_stays_one(where):
    """Such a decay is not taken for 0: outputs and state are NaN from its token on, as token after token."""
    H, P, N, n, bad = 2, 16, 16, 200, 70 if where == "step size" else 0
    g = torch.Generator().manual_seed(9)
    xbc, u, zero = torch.randn(n, H * P + 2 * N, generator=g).bfloat16().cuda(), torch.randn(n, H, generator=g).bfloat16(), torch.zeros(H)
    a_log = zero.clone()
    if where == "A_log":
        a_log[1] = float("nan")
    else:
        u[bad, 1] = float("nan")
    q_start, slot = torch.tensor([0, n], dtype=torch.int32).cuda(), torch.zeros(1, dtype=torch.int32).cuda()
    for form, segments in (("walk", 0), ("chunk", 1), ("chunk", 3)):
        y, state = torch.zeros(n, H, P).cuda(), torch.zeros(1, H, P, N).cuda()
        ops.ssm_scan(y.view(n, -1), xbc, u.cuda(), 0, zero.cuda(), a_log.cuda(), zero.cuda(), state, q_start, slot, 1, max_len=n, form=form, segments=segments, tile=64)
        assert y[bad:, 1].isnan().all() and state[:, 1].isnan().all(), (form, segments)
        assert y[:bad].isfinite().all() and y[:, 0].isfinite().all() and state[:, 0].isfinite().all(), (form, segments)


def _same_kind(got, want, tol):
    """Infinities and NaNs in the same places, and what is finite near."""
    got, fine = got.cpu().double(), want.isfinite()
    return bool((got.isnan() == want.isnan()).all() and (got.isinf() == want.isinf()).all() and (got[want.isinf()] == want[want.isinf()]).all()
                and (got[fine] - want[fine]).norm() <= tol * want[fine].norm())


@pytest.mark.gpu
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.0e38], ids=["inf", "-inf", "nan", "3e38"])
@pytest.mark.parametrize("where", ["x", "B", "C", "dt", "state"])
@pytest.mark.parametrize("bad", [0, 5, 71, 140, 199])
def test_infinities_and_nans_stay_where_the_recurrence_has_them(where, value, bad):
    """A number that is not finite reaches its own and later tokens of its own columns, and no other."""
    H, P, N, n = 2, 72, 24, 200
    g = torch.Generator().manual_seed(11)
    xbc, u, state = torch.randn(n, H * P + 2 * N, generator=g).bfloat16(), torch.randn(n, H, generator=g).bfloat16(), torch.randn(1, H, P, N, generator=g)
    if where == "state":
        state[0, 1, bad % P, 3] = value
    elif where == "dt":
        u[bad, 1] = value
    else:
        xbc[bad, {"x": P + bad % P, "B": H * P + 3, "C": H * P + N + 3}[where]] = value
    vec = torch.randn(3, H, generator=g)
    vec[0] -= 3.0  # small steps: no decay of the whole sequence underflows in float32
    want = _exact(xbc, u, 0, vec[0], vec[1] * 0.1, vec[2], state.clone(), [n], 1)
    if value == 3.0e38:  # what float32 does not hold is infinite there
        want = [w.float().double() for w in want]
    q_start, slot, vec = torch.tensor([0, n], dtype=torch.int32).cuda(), torch.zeros(1, dtype=torch.int32).cuda(), vec.cuda()
    for segments in (1, 3):
        y, st = torch.zeros(n, H * P).cuda(), state.cuda()
        ops.ssm_scan(y, xbc.cuda(), u.cuda(), 0, vec[0], vec[1] * 0.1, vec[2], st, q_start, slot, 1, max_len=n, form="chunk", segments=segments, tile=64)
        if value == 3.0e38:  # (sums of such numbers may leave float32 on the way in one order and not in another: only tokens in front of it are compared)
            assert where == "state" or _same_kind(y[:bad], want[0][:bad], 1e-6)
        else:
            assert _same_kind(y, want[0], 1e-6) and _same_kind(st, want[1], 1e-6)


@pytest.mark.gpu
def test_single_tokens_taken_apart_give_the_same(monkeypatch):
    from dli_b200.cache.pools import LayerCache
    from dli_b200.config.spec import PartSpec
    from dli_b200.engine.batch import StepBatch
    from dli_b200.parts import ssm
    from dli_b200.parts.base import BuildEnv, build_part

    W, H = 64, 4
    params = {"hidden_size": W, "num_heads": H, "head_dim": 32, "state_size": 16, "groups": 2, "conv_taps": 4, "norm_groups": 2, "eps": 1e-6}
    part = build_part("mixer", PartSpec("mamba2", params), BuildEnv(torch.bfloat16, torch.device("cuda")))
    g = torch.Generator().manual_seed(3)
    part.load({name: (torch.randn(decl.shape, generator=g) * 0.2).to(torch.bfloat16 if decl.kind == "matrix" else torch.float32).cuda()
               for name, decl in part.declare().items()})
    lens = [1] * 6 + [40, 25]
    n, S = sum(lens), len(lens)
    x = torch.randn(n, W, generator=g).bfloat16().cuda()
    starts = [(torch.randn((S, *need.shape), generator=g) * 0.3).to(need.dtype).cuda() for need in part.cache_need()]
    q_start = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32).cuda()
    batch = StepBatch(n=n, num_seqs=S, num_single=6, token_ids=None, positions=None, seq_of_token=torch.repeat_interleave(torch.arange(S), torch.tensor(lens)).int().cuda(),
                      q_start=q_start, kv_len=None, state_slot=torch.arange(S, dtype=torch.int32, device="cuda"), logit_rows=None, groups=[], max_q_len=40)
    got = []
    for apart in (0, 6):
        monkeypatch.setattr(ssm, "scan_singles_apart", lambda *a: apart)
        cache = LayerCache(states=tuple(s.clone() for s in starts))
        got.append([part.forward(x, batch, cache), *cache.states])
    for a, b in zip(*got):  # bfloat16 outputs of float32 sums that differ in their order; float32 states
        assert (a.float() - b.float()).norm() <= (1e-2 if a.dtype == torch.bfloat16 else 1e-5) * b.float().norm()


@pytest.mark.gpu
def test_read_outs_off_an_8_byte_boundary_are_walked():
    H, P, N, n = 2, 16, 16, 100
    g = torch.Generator().manual_seed(3)
    xbc, u, state = torch.randn(n, H * P + 2 * N, generator=g).bfloat16(), torch.randn(n, H, generator=g).bfloat16(), torch.randn(1, H, P, N, generator=g)
    zero = torch.zeros(H)
    want = _exact(xbc, u, 0, zero, zero, zero, state.clone(), [n], 1)
    room, st = torch.zeros(n * H * P + 1).cuda(), state.cuda()
    y = room[1:].view(n, H * P)
    ops.ssm_scan(y, xbc.cuda(), u.cuda(), 0, zero.cuda(), zero.cuda(), zero.cuda(), st, torch.tensor([0, n], dtype=torch.int32).cuda(), torch.zeros(1, dtype=torch.int32).cuda(), 1,
                 max_len=n)
    assert all((a.cpu().double() - b).norm() <= 2e-6 * b.norm() for a, b in ((y, want[0]), (st, want[1]))) and room[0] == 0


@pytest.mark.gpu
def test_a_tile_may_be_replayed_from_a_graph():
    H, P, N, lens = 2, 64, 64, [1, 200]
    xbc, u = torch.randn(201, H * P + 2 * N).bfloat16().cuda(), torch.randn(201, H).bfloat16().cuda()
    one, q_start, slot = torch.zeros(H).cuda(), torch.tensor([0, 1, 201], dtype=torch.int32).cuda(), torch.tensor([0, 1], dtype=torch.int32).cuda()
    state = torch.zeros(2, H, P, N).cuda()
    want, got = torch.empty(201, H * P).cuda(), torch.empty(201, H * P).cuda()
    ops.ssm_scan(want, xbc, u, 0, one, one, one, state, q_start, slot, 1, max_len=200)
    end = state.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.ssm_scan(got, xbc, u, 0, one, one, one, state, q_start, slot, 1, max_len=200)
    state.zero_()
    graph.replay()
    assert torch.equal(got, want) and torch.equal(state, end)


@pytest.mark.gpu
@pytest.mark.parametrize("tile", [64, 128])
@pytest.mark.parametrize("segments", [1, 3])
def test_a_recorded_step_takes_other_sequences(segments, tile):
    """Recorded once and replayed with other sequences: empty ones in the middle and at the end, and rows behind the last token that belong to none."""
    H, P, N, rows, steps = 2, 24, 32, 210, ([1, 63, 65, 0, 71], [0, 200, 1, 9, 0], [64, 0, 0, 2, 128], [0, 0, 0, 0, 0])
    S, g = len(steps[0]), torch.Generator().manual_seed(19)
    xbc, u, start = torch.randn(rows, H * P + 2 * N, generator=g).bfloat16(), torch.randn(rows, H, generator=g).bfloat16(), torch.randn(S, H, P, N, generator=g)
    vec = torch.randn(3, H, generator=g)
    x, q_start, slot = [t.cuda() for t in (xbc, u, *vec)], torch.zeros(S + 1, dtype=torch.int32).cuda(), torch.arange(S, dtype=torch.int32).cuda()
    y, state = torch.zeros(rows, H * P).cuda(), start.cuda()

    def run():
        ops.ssm_scan(y, x[0], x[1], 0, x[2], x[3], x[4], state, q_start, slot, 1, max_len=rows, form="chunk", segments=segments, tile=tile)

    run()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
    for lens in steps:
        n, order = sum(lens), torch.randperm(S, generator=g)
        q_start.copy_(torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()])), slot.copy_(order.int()), state.copy_(start), y.fill_(7.0)
        graph.replay()
        first = start[order]
        want = _exact(xbc, u, 0, *vec, first.clone(), lens, 1) if n else (torch.zeros(0, H * P, dtype=torch.float64), first.double())
        assert all((a.double() - b).norm() <= 5.4e-6 * b.norm() for a, b in ((y[:n].cpu(), want[0]), (state.cpu()[order], want[1]))) and (y[n:] == 7.0).all(), lens


def test_which_form_serves_a_step():
    form, bf, f32 = ops.ssm_scan_form, torch.bfloat16, torch.float32
    assert form(bf, 64, 128, 17) == "chunk" and form(bf, 8, 8, 1 << 30) == "chunk"
    assert form(bf, 64, 128, 16) == "walk"  # a decode step, or a short portion
    assert form(f32, 64, 128, 4096) == "walk"
    assert form(bf, 64, 136, 4096) == form(bf, 20, 16, 4096) == form(bf, 64, 10, 4096) == "walk"  # larger states; rows that are not whole 16-byte runs
    assert form(bf, 64, 128, 4096, aligned=False) == "walk"
