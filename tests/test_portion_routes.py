"""Which kernels the host gives a step's portions to: the lines between two kernels lie where measurements of both put them.  No GPU needed."""

import types

import pytest
import torch

from dli_b200.kernels import attention, ops
from dli_b200.parts import ssm


@pytest.mark.parametrize("portion,step,tiles", [(64, 64, False), (2, 2, False), (65, 65, True), (4096, 4096, True), (64, 3000, False), (3000, 3000, True), (0, 64, False),
                                                (0, 65, True), (0, 0, True)])
def test_portions_over_one_pool_of_rows(portion, step, tiles):
    """One key tile of the mma.sync kernel: that kernel.  What the step does not say of its portions, its longest sequence bounds; 0: not known."""
    assert attention.portions_pay_for_tiles_of_rows(types.SimpleNamespace(max_kv_len_portion=portion, max_kv_len=step)) == tiles


@pytest.mark.parametrize("portions,singles,context,apart", [
    ([(2, 0)], 0, 0, False), ([(2, 300)], 0, 0, False), ([(64, 0)], 0, 0, True), ([(300, 0)], 0, 0, True), ([(1024, 0)], 0, 0, True), ([(128, 3000)], 0, 0, True),
    ([(16, 0)], 24, 200, False), ([(3, 200)] * 8, 64, 300, False), ([(512, 512)], 24, 200, True), ([(16, 0)], 24, 3000, True), ([(128, 0)], 64, 2000, False),
    ([(128, 3000)], 64, 2000, True), ([(1535, 1024)], 9, 1500, True)])
def test_portions_of_differential_attention(portions, singles, context, apart):
    """Few tokens beside single tokens go with them in one launch; portions that make up a launch go to the tcgen05 kernel."""
    longest = max(q + before for q, before in portions)
    batch = types.SimpleNamespace(num_single=singles, num_seqs=singles + len(portions), max_q_len=max(q for q, _ in portions), max_kv_len=max(longest, context), max_kv_len_single=context, max_kv_len_portion=longest)
    assert attention.diff_portions_apart(batch, singles + sum(q for q, _ in portions), 16, 4, None, 0) == apart


@pytest.mark.parametrize("kind,heads,d,singles,portions,route", [
    ("channel", 16, 128, 0, [2048], "tiles"), ("channel", 16, 128, 0, [48], "tiles"), ("channel", 8, 128, 0, [33], "walk"), ("channel", 4, 64, 0, [33], "walk"),
    ("channel", 16, 128, 0, [33] * 32, "walk"), ("channel", 16, 64, 0, [100] * 32, "walk"), ("channel", 8, 128, 3, [33], "walk"), ("channel", 16, 128, 8, [64], "walk"),
    ("channel", 16, 128, 8, [100], "apart"), ("channel", 16, 128, 24, [300], "apart"), ("channel", 4, 64, 64, [33], "walk"), ("channel", 16, 128, 64, [], "walk"),
    ("bonus", 16, 64, 0, [250, 251], "tiles"), ("bonus", 64, 64, 0, [33] * 32, "walk"), ("bonus", 64, 64, 0, [200] * 16, "walk"), ("bonus", 16, 64, 4, [33], "walk"),
    ("bonus", 16, 64, 0, [1500], "tiles"), ("bonus", 16, 64, 24, [300], "tiles"), ("head", 16, 128, 0, [33], "tiles"), ("head", 16, 128, 24, [64], "apart")])
def test_steps_of_the_recurrences(kind, heads, d, singles, portions, route):
    """Every kind by its own costs: short portions, and many portions of wide models, are walked where that was measured to be faster."""
    batch = types.SimpleNamespace(num_single=singles, num_seqs=singles + len(portions), n=singles + sum(portions), max_q_len=max(portions, default=1))
    if kind != "bonus" and ssm.singles_apart(batch, d, d, heads, True, kind):
        assert route == "apart"
    else:
        assert ops.recurrence_form(d, d, batch.max_q_len, batch.n, batch.num_seqs, heads, True, kind, singles) == route


@pytest.mark.parametrize("heads,singles,portions,apart", [(64, 24, [17], 24), (64, 64, [64], 64), (128, 4, [33], 4), (64, 4, [33], 0), (64, 8, [17], 0), (64, 16, [300], 0),
                                                          (64, 24, [16], 0), (64, 24, [], 0), (128, 0, [33] * 16, 0), (128, 3, [33] * 16, 0), (16, 24, [33], 0)])
def test_single_tokens_beside_a_scan(heads, singles, portions, apart):
    """They are walked by themselves where their tiles would queue behind one another while portions of one tile wait for them."""
    batch = types.SimpleNamespace(num_single=singles, num_seqs=singles + len(portions), n=singles + sum(portions), max_q_len=max(portions, default=1))
    assert ssm.scan_singles_apart(batch, 64, 128, heads, torch.bfloat16) == apart
    assert ssm.scan_singles_apart(batch, 64, 128, heads, torch.float32) == 0


@pytest.mark.parametrize("portions,singles,context,window,beside", [
    ([(1535, 1024)], 9, 1500, 1024, True), ([(1535, 1024)], 9, 1500, None, True), ([(1535, 0)], 9, 1500, None, False), ([(1535, 0)], 9, 300, None, True),
    ([(1024, 0)], 4, 900, None, True), ([(1024, 0)], 4, 3000, None, False), ([(1535, 1024)], 64, 1500, 1024, False), ([(0, 0)], 4, 100, None, False)])
def test_single_tokens_beside_portions_of_differential_attention(portions, singles, context, window, beside, monkeypatch):
    """In the portions' launch where its last wave has places for all and they see little more than its last CTAs; a recorded step keeps them apart."""
    monkeypatch.setattr(attention, "sm_count", lambda: 148)
    lens, starts = [1] * singles + [q for q, _ in portions], [context - 1] * singles + [before for _, before in portions]
    batch = types.SimpleNamespace(num_single=singles, num_seqs=len(lens), q_lens=lens, starts=starts, max_kv_len_single=context, max_kv_len=max(q + b for q, b in zip(lens, starts)),
                                  max_kv_len_portion=max(q + b for q, b in portions))
    assert attention.diff_singles_beside(batch, 16, 4, window, 16 if window else 0) == beside


@pytest.mark.parametrize("portions,singles,context,nh,nkv,beside", [([(200, 0)], 1, 8000, 8, 2, False), ([(200, 1024)], 40, 8000, 8, 2, False), ([(500, 1024)], 1, 8000, 32, 8, False),
                                                                  ([(200, 1024)], 2, 3000, 32, 8, False), ([(500, 512)], 1, 700, 16, 4, True)])
def test_long_single_tokens_stay_apart_whatever_the_step_says_of_its_portions(portions, singles, context, nh, nkv, beside, monkeypatch):
    """A step that names only its longest sequence: the portions' keys follow from their lengths, not from the single tokens' context."""
    monkeypatch.setattr(attention, "sm_count", lambda: 148)
    lens, starts = [1] * singles + [q for q, _ in portions], [context - 1] * singles + [before for _, before in portions]
    batch = types.SimpleNamespace(num_single=singles, num_seqs=len(lens), q_lens=lens, starts=starts, max_kv_len_single=context, max_kv_len=max(context, *(q + b for q, b in portions)))
    assert attention.diff_singles_beside(batch, nh, nkv, None, 0) == beside


@pytest.mark.parametrize("heads,P,N,singles,portions,tile", [
    (64, 64, 128, 0, [33], 128), (64, 64, 128, 0, [32], 64), (64, 64, 128, 0, [1000, 666, 1335], 128), (32, 128, 64, 0, [13, 55, 58, 58], 64), (128, 64, 128, 0, [25, 18, 11, 32, 36], 64),
    (128, 32, 64, 0, [73, 66, 51, 63, 43], 64), (32, 128, 32, 24, [151, 153, 159], 64), (32, 64, 64, 4, [35, 24, 44, 49], 64), (64, 64, 128, 24, [100], 128), (32, 64, 64, 0, [1177], 64),
    (32, 64, 64, 0, [616], 128), (32, 64, 64, 0, [3057], 128), (8, 64, 32, 3, [1330], 64), (8, 64, 128, 0, [1330], 128), (64, 64, 40, 0, [600], 64), (64, 64, 16, 0, [600], 64)])
def test_tiles_of_the_scan(heads, P, N, singles, portions, tile):
    """Tiles of 128 tokens where their CTAs, each with an SM to itself, do not queue with short portions."""
    n, count = singles + sum(portions), singles + len(portions)
    assert ops.ssm_tile(heads, P, N, n, count, (len(portions), sum(portions) / len(portions)), max(portions)) == tile


@pytest.mark.parametrize("heads,d,singles,portions,tile", [
    (16, 128, 0, [48], 64), (16, 128, 7, [600], 128), (16, 128, 0, [28] * 5 + [49], 64), (16, 128, 0, [89] * 6, 128), (16, 128, 16, [30, 60], 128), (32, 64, 0, [54, 69, 21, 82, 30], 64),
    (32, 64, 0, [200] * 5, 128), (32, 32, 0, [100] * 8, 64), (16, 32, 0, [100], 128), (16, 64, 48, [37, 50], 128)])
def test_tiles_of_the_matrix_memory(heads, d, singles, portions, tile):
    n, count = singles + sum(portions), singles + len(portions)
    assert ops.matrix_memory_tile(heads, d, d, n, count, (len(portions), sum(portions) / len(portions)), max(portions)) == tile


def test_what_a_step_says_of_its_portions():
    """As it is; a recorded one (its portions have no lengths yet, one of its sequences stays empty) the tokens of all together; without word the longest bounds the others."""
    start = types.SimpleNamespace(is_cuda=True)
    assert ssm.tile_hint(types.SimpleNamespace(q_lens=[1, 1, 30, 10], num_single=2, n=42, q_start=start)) == {"portions": (2, 20.0)}
    assert ssm.tile_hint(types.SimpleNamespace(q_lens=[1, 1, 0, 0, 0], num_single=2, n=66, q_start=start)) == {"portions": (2, 32.0)}
    assert ssm.tile_hint(types.SimpleNamespace(num_single=0, n=42, q_start=start)) == {}
    assert ops.ssm_tile(64, 64, 128, 600, 1, None, 1 << 30) == 128 and ops.ssm_tile(64, 64, 128, 100, 10, None, 40) == 64
