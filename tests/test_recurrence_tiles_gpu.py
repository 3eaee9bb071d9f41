"""The delta rules and the token-shift recurrence over tiles of tokens (csrc/recurrence_tiles.cu) against the recurrences in float64, at the edges of
their tiles, blocks and column groups; and which kernels serve which step."""

import types

import pytest
import torch

from dli_b200.kernels import ops
from dli_b200.parts import ssm


def _unit(v):
    return v / torch.sqrt((v * v).sum(-1, keepdim=True) + 1e-6)


def _starts(lens):
    return torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32)


def _delta(channel, qkv, u, a, dt_bias, a_log, state, lens, G):
    """u: betas' columns 1 .. heads, then the decays' ones of the rule with a decay per head."""
    S, H, dv, d = state.shape
    n, x = qkv.shape[0], qkv.double()
    q = (_unit(x[:, : G * d].view(n, G, d)) * d**-0.5).repeat_interleave(H // G, 1)
    k = _unit(x[:, G * d : 2 * G * d].view(n, G, d)).repeat_interleave(H // G, 1)
    v, beta = x[:, 2 * G * d :].view(n, H, dv), torch.sigmoid(u[:, 1 : 1 + H].double())
    raw = (a.double() + dt_bias.double()).view(n, H, d) if channel else (u[:, 1 + H : 1 + 2 * H].double() + dt_bias.double())[..., None]
    keep = torch.exp(-torch.exp(a_log.double())[:, None] * torch.nn.functional.softplus(raw))
    state, out, t0 = state.double(), [], 0
    for s, count in enumerate(lens):
        X = state[s]
        for t in range(t0, t0 + count):
            X = X * keep[t, :, None, :]
            X = X + (beta[t, :, None] * (v[t] - (X @ k[t, :, :, None])[..., 0]))[:, :, None] * k[t, :, None, :]
            out.append((X @ q[t, :, :, None])[..., 0].reshape(-1))
        state[s], t0 = X, t0 + count
    return torch.stack(out), state


def _bonus(rkvg, wz, w0, bonus, state, lens):
    S, H, _, d = state.shape
    n = wz.shape[0]
    r, k, v = (rkvg[i].double().view(n, H, d) for i in range(3))
    keep = torch.exp(-torch.exp(wz.double() + w0.double())).view(n, H, d)
    state, out, t0 = state.double(), [], 0
    for s, count in enumerate(lens):
        X = state[s]
        for t in range(t0, t0 + count):
            kv = v[t, :, :, None] * k[t, :, None, :]
            out.append(((X + kv * bonus.double()[:, None, :]) @ r[t, :, :, None])[..., 0].reshape(-1))
            X = X * keep[t, :, None, :] + kv
        state[s], t0 = X, t0 + count
    return torch.stack(out), state


def _check(run, want, shape, state):
    """Both forms from the same start.  Float32, token after token: some four roundings of 2^-24 a token that add up at random over at most 200 tokens, 1.7e-6,
    and twice that for scatter.  The tiles are no worse than the walk by more than the scatter between two orders of summation."""
    S = state.shape[0]
    slot = torch.arange(S - 1, -1, -1, dtype=torch.int32, device="cuda")  # slots in another order than the sequences
    errors = {}
    for form in ("walk", "tiles"):
        o, st = torch.full(shape, float("nan"), device="cuda"), state.flip(0).cuda()
        run(o, st, slot, form)
        errors[form] = [float((x.cpu().double() - y).norm() / y.norm()) for x, y in ((o, want[0]), (st.flip(0), want[1]))]
    assert all(e <= 3.4e-6 for form in errors.values() for e in form), errors
    assert all(e <= max(2 * w, 5e-7) for e, w in zip(errors["tiles"], errors["walk"])), errors
    assert ops.device_wait_errors() == {}


SHAPES = [(2, 1, 128, 128, [1, 63, 64, 65]), (4, 2, 64, 64, [130, 17]), (2, 2, 40, 24, [200, 2]), (3, 1, 128, 16, [16, 33]), (2, 1, 13, 9, [70]), (40, 20, 128, 128, [65])]


@pytest.mark.gpu
@pytest.mark.parametrize("decay", [-6.0, 0.0, 30.0], ids=["long_memory", "short_memory", "no_memory"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("channel", [False, True], ids=["decay_per_head", "decay_per_channel"])
@pytest.mark.parametrize("H,G,d,dv,lens", SHAPES)
def test_delta_rules(H, G, d, dv, lens, channel, dtype, decay):
    g = torch.Generator().manual_seed(H * 100 + d + dv)
    n = sum(lens)
    qkv, u = torch.randn(n, 2 * G * d + H * dv, generator=g).to(dtype), torch.randn(n, 2 * H + 3, generator=g).to(dtype)
    a, a_log = torch.randn(n, H * d, generator=g).to(dtype), torch.rand(H, generator=g)
    dt_bias = torch.randn(H * d if channel else H, generator=g) + decay
    state = torch.randn(len(lens), H, dv, d, generator=g) * 0.3
    want = _delta(channel, qkv, u, a, dt_bias, a_log, state, lens, G)
    q_start, seq = _starts(lens).cuda(), torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).int().cuda()
    x = [t.cuda() for t in (qkv, u, a, dt_bias, a_log)]

    def run(o, st, slot, form):
        if channel:
            ops.channel_delta_scan(o, x[0], x[1], 1, x[2], x[3], x[4], st, q_start, slot, G, 1e-6, max_len=max(lens), form=form)
        else:
            ops.delta_rule_scan(o, x[0], x[1], 1, 1 + H, x[3], x[4], st, seq, q_start, slot, G, d, 1e-6, max_len=max(lens), form=form)

    _check(run, want, (n, H * dv), state)


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [-5.0, 0.0, 5.0], ids=["long_memory", "short_memory", "no_memory"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H,d,lens", [(2, 64, [1, 63, 64, 65]), (2, 128, [130, 17]), (3, 24, [100]), (1, 9, [33, 1, 70]), (40, 64, [65])])
def test_bonus(H, d, lens, dtype, shift):
    g = torch.Generator().manual_seed(H * 100 + d)
    n = sum(lens)
    rkvg, wz = torch.randn(4, n, H * d, generator=g).to(dtype), torch.randn(n, H * d, generator=g).to(dtype)
    w0, bonus, state = torch.randn(H * d, generator=g) + shift, torch.randn(H, d, generator=g), torch.randn(len(lens), H, d, d, generator=g)
    want = _bonus(rkvg, wz, w0, bonus, state, lens)
    q_start, x = _starts(lens).cuda(), [t.cuda() for t in (rkvg, wz, w0, bonus)]
    _check(lambda o, st, slot, form: ops.shift_decay_scan(o, x[0], x[1], x[2], "bonus", x[3], st, q_start, slot, max_len=max(lens), form=form), want, (n, H * d), state)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("channel", [False, True], ids=["decay_per_head", "decay_per_channel"])
def test_a_gate_that_is_not_a_number_stays_one(channel, dtype):
    """Such a decay is not taken for 0: outputs and state are NaN from its token on, as token after token."""
    H, d, n, bad = 2, 16, 150, 70
    g = torch.Generator().manual_seed(9)
    qkv, u, a = (torch.randn(n, c, generator=g).to(dtype) for c in (3 * H * d, 2 * H, H * d))
    (a if channel else u)[bad, d if channel else H + 1] = float("nan")  # of head 1
    q_start, slot, seq = torch.tensor([0, n], dtype=torch.int32).cuda(), torch.zeros(1, dtype=torch.int32).cuda(), torch.zeros(n, dtype=torch.int32).cuda()
    zero, qkv, u, a = torch.zeros(H).cuda(), qkv.cuda(), u.cuda(), a.cuda()
    for form in ("walk", "tiles"):
        o, state = torch.zeros(n, H, d).cuda(), torch.full((1, H, d, d), 0.1).cuda()
        if channel:
            ops.channel_delta_scan(o.view(n, -1), qkv, u, 0, a, torch.zeros(H * d).cuda(), zero, state, q_start, slot, H, 1e-6, max_len=n, form=form)
        else:
            ops.delta_rule_scan(o.view(n, -1), qkv, u, 0, H, zero, zero, state, seq, q_start, slot, H, d, 1e-6, max_len=n, form=form)
        assert o[bad:, 1].isnan().all() and state[:, 1].isnan().all(), form
        assert o[:64].isfinite().all() and o[:, 0].isfinite().all() and state[:, 0].isfinite().all(), form


def _same_kind(got, want, tol):
    """Infinities and NaNs in the same places, and what is finite near."""
    got, fine = got.cpu().double(), want.isfinite()
    return bool((got.isnan() == want.isnan()).all() and (got.isinf() == want.isinf()).all() and (got[want.isinf()] == want[want.isinf()]).all()
                and (got[fine] - want[fine]).norm() <= tol * want[fine].norm())


@pytest.mark.gpu
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")], ids=["inf", "-inf", "nan"])
@pytest.mark.parametrize("where", ["q", "k", "v", "gate", "beta", "state"])
@pytest.mark.parametrize("bad", [0, 5, 71, 149])
@pytest.mark.parametrize("kind,dtype,d,dv", [("head", torch.bfloat16, 24, 40), ("head", torch.float32, 24, 17), ("channel", torch.bfloat16, 128, 20), ("channel", torch.float32, 30, 8),
                                             ("bonus", torch.bfloat16, 40, 40), ("bonus", torch.float32, 9, 9)])
def test_infinities_and_nans_stay_where_the_recurrence_has_them(kind, dtype, d, dv, where, value, bad):
    """A number that is not finite reaches its own and later tokens, of a value or a state its own columns only, and no other."""
    H, n = 2, 150
    if kind == "bonus" and where == "beta":
        pytest.skip("no beta")
    g = torch.Generator().manual_seed(13)
    qkv = torch.randn(4, n, H * d, generator=g) if kind == "bonus" else torch.randn(n, 2 * H * d + H * dv, generator=g)
    u, a, state = torch.randn(n, 2 * H + 1, generator=g), torch.randn(n, H * d, generator=g), torch.randn(1, H, dv, d, generator=g)
    bias, a_log, bonus = torch.randn(H if kind == "head" else H * d, generator=g) - 4.0, torch.zeros(H), torch.randn(H, d, generator=g)
    if where == "state":
        state[0, 1, bad % dv, 3] = value
    elif where == "beta":
        u[bad, 2] = value
    elif where == "gate":
        (u if kind == "head" else a)[bad, 1 + H + 1 if kind == "head" else d + 3] = value
    elif kind == "bonus":
        qkv["qkv".index(where), bad, d + bad % d] = value
    else:
        qkv[bad, {"q": d + 3, "k": H * d + d + 3, "v": 2 * H * d + dv + bad % dv}[where]] = value
    qkv, u, a = qkv.to(dtype), u.to(dtype), a.to(dtype)
    want = _bonus(qkv, a, bias, bonus, state, [n]) if kind == "bonus" else _delta(kind == "channel", qkv, u, a, bias, a_log, state, [n], H)
    q_start, slot, seq = torch.tensor([0, n], dtype=torch.int32).cuda(), torch.zeros(1, dtype=torch.int32).cuda(), torch.zeros(n, dtype=torch.int32).cuda()
    o, st, x = torch.zeros(n, H * dv).cuda(), state.cuda(), [t.cuda() for t in (qkv, u, a, bias, a_log, bonus)]
    if kind == "bonus":
        ops.shift_decay_scan(o, x[0], x[2], x[3], "bonus", x[5], st, q_start, slot, max_len=n, form="tiles")
    elif kind == "channel":
        ops.channel_delta_scan(o, x[0], x[1], 1, x[2], x[3], x[4], st, q_start, slot, H, 1e-6, max_len=n, form="tiles")
    else:
        ops.delta_rule_scan(o, x[0], x[1], 1, 1 + H, x[3], x[4], st, seq, q_start, slot, H, d, 1e-6, max_len=n, form="tiles")
    assert _same_kind(o, want[0], 2e-6) and _same_kind(st, want[1], 2e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("channel,dtype", [(False, torch.bfloat16), (False, torch.float32), (True, torch.bfloat16)])
def test_read_outs_off_an_8_byte_boundary(channel, dtype):
    H, d, n = 2, 16, 100
    g = torch.Generator().manual_seed(3)
    qkv, u, a = (torch.randn(n, c, generator=g).to(dtype) for c in (3 * H * d, 2 * H + 1, H * d))
    bias, a_log, state = torch.randn(H * d if channel else H, generator=g), torch.zeros(H), torch.randn(1, H, d, d, generator=g)
    want = _delta(channel, qkv, u, a, bias, a_log, state, [n], H)
    room, st = torch.zeros(n * H * d + 1).cuda(), state.cuda()
    o, q_start, slot = room[1:].view(n, H * d), torch.tensor([0, n], dtype=torch.int32).cuda(), torch.zeros(1, dtype=torch.int32).cuda()
    qkv, u, a, bias, a_log = (x.cuda() for x in (qkv, u, a, bias, a_log))
    if channel:
        ops.channel_delta_scan(o, qkv, u, 1, a, bias, a_log, st, q_start, slot, H, 1e-6, max_len=n, form="tiles")
    else:
        ops.delta_rule_scan(o, qkv, u, 1, 1 + H, bias, a_log, st, torch.zeros(n, dtype=torch.int32).cuda(), q_start, slot, H, d, 1e-6, max_len=n, form="tiles")
    assert all((x.cpu().double() - y).norm() <= 2e-6 * y.norm() for x, y in ((o, want[0]), (st, want[1]))) and room[0] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("kind,dtype,least", [("head", torch.bfloat16, 140e3), ("channel", torch.bfloat16, 210e3), ("bonus", torch.bfloat16, 158e3), ("head", torch.float32, 210e3)])
def test_a_step_whose_tiles_outgrow_the_scratch_goes_in_passes(kind, dtype, least, monkeypatch):
    """The scratch is that of the tiles' kind and no larger than its limit; the state between two passes waits in its slot, so nothing changes."""
    H, d, lens = 4, 128, [1, 200, 0, 64, 0, 130]
    g, n = torch.Generator().manual_seed(17), sum(lens)
    qkv = torch.randn(4, n, H * d, generator=g) if kind == "bonus" else torch.randn(n, 3 * H * d, generator=g)
    u, a = torch.randn(n, 2 * H, generator=g).to(dtype).cuda(), torch.randn(n, H * d, generator=g).to(dtype).cuda()
    qkv, start = qkv.to(dtype).cuda(), torch.randn(len(lens), H, d, d, generator=g).cuda()
    bias, a_log, bonus = (torch.randn(H if kind == "head" else H * d, generator=g) - 3.0).cuda(), torch.zeros(H).cuda(), torch.randn(H, d, generator=g).cuda()
    q_start, slot = _starts(lens).cuda(), torch.arange(len(lens), dtype=torch.int32, device="cuda")
    seq, got, calls = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).int().cuda(), [], []
    for limit in (1 << 30, 1):
        monkeypatch.setattr(ops, "TILES_SCRATCH_LIMIT", limit)
        o, state = torch.zeros(n, H * d).cuda(), start.clone()
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before, launched = torch.cuda.memory_allocated(), ops.launch_count
        if kind == "bonus":
            ops.shift_decay_scan(o, qkv, a, bias, "bonus", bonus, state, q_start, slot, max_len=200, form="tiles")
        elif kind == "channel":
            ops.channel_delta_scan(o, qkv, u, 0, a, bias, a_log, state, q_start, slot, H, 1e-6, max_len=200, form="tiles")
        else:
            ops.delta_rule_scan(o, qkv, u, 0, H, bias, a_log, state, seq, q_start, slot, H, d, 1e-6, max_len=200, form="tiles")
        places = n // 64 + len(lens) + 1
        assert torch.cuda.max_memory_allocated() - before <= (places if limit > 1 else 1) * H * least + (1 << 20)  # (the allocator may hand out a block up to 1 MiB larger)
        calls.append(ops.launch_count - launched)
        got.append((o, state))
    assert calls[1] == places * calls[0] and all(torch.equal(x, y) for x, y in zip(*got))


@pytest.mark.gpu
@pytest.mark.parametrize("kind,dtype", [("head", torch.bfloat16), ("head", torch.float32), ("channel", torch.bfloat16), ("bonus", torch.bfloat16)])
def test_a_recorded_step_takes_other_sequences(kind, dtype):
    """Recorded once and replayed with other sequences: empty ones in the middle and at the end, and rows behind the last token that belong to none."""
    H, d, rows, steps = 2, 64, 210, ([1, 63, 65, 0, 71], [0, 130, 1, 64, 0], [64, 0, 0, 2, 128], [0, 0, 0, 0, 0])
    S, g = len(steps[0]), torch.Generator().manual_seed(19)
    qkv = torch.randn(4, rows, H * d, generator=g) if kind == "bonus" else torch.randn(rows, 3 * H * d, generator=g)
    qkv, u, a = qkv.to(dtype), torch.randn(rows, 2 * H + 1, generator=g).to(dtype), torch.randn(rows, H * d, generator=g).to(dtype)
    bias, a_log, bonus = torch.randn(H if kind == "head" else H * d, generator=g) - 3.0, torch.zeros(H), torch.randn(H, d, generator=g)
    start, x = torch.randn(S, H, d, d, generator=g), [t.cuda() for t in (qkv, u, a, bias, a_log, bonus)]
    q_start, slot, o, state = _starts(steps[0]).cuda(), torch.arange(S, dtype=torch.int32).cuda(), torch.zeros(rows, H * d).cuda(), start.cuda()
    seq = torch.zeros(rows, dtype=torch.int32).cuda()

    def run():
        if kind == "bonus":
            ops.shift_decay_scan(o, x[0], x[2], x[3], "bonus", x[5], state, q_start, slot, max_len=rows, form="tiles")
        elif kind == "channel":
            ops.channel_delta_scan(o, x[0], x[1], 1, x[2], x[3], x[4], state, q_start, slot, H, 1e-6, max_len=rows, form="tiles")
        else:
            ops.delta_rule_scan(o, x[0], x[1], 1, 1 + H, x[3], x[4], state, seq, q_start, slot, H, d, 1e-6, max_len=rows, form="tiles")

    run()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
    for lens in steps:
        n, order = sum(lens), torch.randperm(S, generator=g)
        q_start.copy_(_starts(lens)), slot.copy_(order.int()), state.copy_(start), o.fill_(7.0)
        graph.replay()
        first = start[order]
        if n == 0:
            want = torch.zeros(0, H * d, dtype=torch.float64), first.double()
        elif kind == "bonus":
            want = _bonus(qkv[:, :n], a[:n], bias, bonus, first, lens)
        else:
            want = _delta(kind == "channel", qkv[:n], u[:n], a[:n], bias, a_log, first, lens, H)
        assert all((p.double() - w).norm() <= 3.4e-6 * w.norm() for p, w in ((o[:n].cpu(), want[0]), (state.cpu()[order], want[1]))) and (o[n:] == 7.0).all(), lens


def test_which_form_serves_a_step():
    form = ops.recurrence_form
    assert form(128, 128, 2048, 2048, 1, 16) == form(64, 64, 4096, 4096, 1, 16) == form(128, 128, 2100, 3500, 2, 16) == form(128, 128, 1 << 30, 2048, 1, 32) == "tiles"
    assert form(128, 128, 1, 64, 64, 16) == form(128, 128, 32, 32, 1, 16) == "walk"  # decode steps, short portions
    assert form(136, 128, 2048, 2048, 1, 16) == form(128, 136, 2048, 2048, 1, 16) == "walk"  # larger heads
    assert form(128, 128, 100, 124, 25, 16) == "walk"  # a single portion does not pay for a tile of every single token
    assert form(128, 128, 2048, 2048, 1, 16, on_gpu=False) == "walk"


def test_when_single_tokens_are_taken_apart():
    def apart(singles, portions, tokens, longest):
        batch = types.SimpleNamespace(num_single=singles, num_seqs=singles + portions, n=singles + tokens, max_q_len=longest)
        return ssm.singles_apart(batch, 128, 128, 16, True)

    assert apart(24, 1, 600, 600) == 24 and apart(4, 2, 300, 200) == 4
    assert apart(3, 1, 600, 600) == 0  # a few ride along
    assert apart(24, 0, 0, 1) == 0 and apart(24, 1, 20, 20) == 0  # nothing, or nothing long enough, beside them


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["gated_delta", "channel_delta"])
def test_single_tokens_taken_apart_give_the_same(kind, monkeypatch):
    from dli_b200.cache.pools import LayerCache
    from dli_b200.config.spec import PartSpec
    from dli_b200.engine.batch import StepBatch
    from dli_b200.parts.base import BuildEnv, build_part

    W, H, G, d = 64, 4, 2, 32
    params = {"hidden_size": W, "num_heads": H, "num_kv_heads": G, "head_dim": d, "value_dim": d, "conv_taps": 4, "eps": 1e-6, "decay_rank": 8, "gate_rank": 8}
    part = build_part("mixer", PartSpec(kind, params), BuildEnv(torch.bfloat16, torch.device("cuda")))
    g = torch.Generator().manual_seed(3)
    part.load({name: (torch.randn(decl.shape, generator=g) * 0.2).to(torch.bfloat16 if decl.kind == "matrix" else torch.float32).cuda()
               for name, decl in part.declare().items()})
    lens = [1] * 6 + [130, 40]
    n, S = sum(lens), len(lens)
    x = torch.randn(n, W, generator=g).bfloat16().cuda()
    starts = [(torch.randn((S, *need.shape), generator=g) * 0.3).to(need.dtype).cuda() for need in part.cache_need()]
    q_start = _starts(lens).cuda()
    batch = StepBatch(n=n, num_seqs=S, num_single=6, token_ids=None, positions=None, seq_of_token=torch.repeat_interleave(torch.arange(S), torch.tensor(lens)).int().cuda(),
                      q_start=q_start, kv_len=None, state_slot=torch.arange(S, dtype=torch.int32, device="cuda"), logit_rows=None, groups=[], max_q_len=130)
    got = []
    for limit in (4, 100):
        monkeypatch.setattr(ssm, "SINGLES_APART", limit)
        cache = LayerCache(states=tuple(s.clone() for s in starts))
        got.append([part.forward(x, batch, cache), *cache.states])
    for a, b in zip(*got):  # bfloat16 outputs of float32 sums that differ in their order; float32 states
        assert (a.float() - b.float()).norm() <= (1e-2 if a.dtype == torch.bfloat16 else 1e-5) * b.float().norm()
