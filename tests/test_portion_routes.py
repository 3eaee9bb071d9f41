"""Which kernels the host gives a step's portions to: the lines between two kernels lie where measurements of both put them.  No GPU needed."""

import types

import pytest

from dli_b200.kernels import attention


@pytest.mark.parametrize("portion,step,tiles", [(64, 64, False), (2, 2, False), (65, 65, True), (4096, 4096, True), (64, 3000, False), (3000, 3000, True), (0, 64, False),
                                                (0, 65, True), (0, 0, True)])
def test_portions_over_one_pool_of_rows(portion, step, tiles):
    """One key tile of the mma.sync kernel: that kernel.  What the step does not say of its portions, its longest sequence bounds; 0: not known."""
    assert attention.portions_pay_for_tiles_of_rows(types.SimpleNamespace(max_kv_len_portion=portion, max_kv_len=step)) == tiles
