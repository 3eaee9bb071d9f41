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
