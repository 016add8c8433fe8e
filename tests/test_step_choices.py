"""Rules by which a step picks a kernel, on either side of their lines, without a GPU."""
import pytest

from cpp_minilamma_b200.parts.state_mixers import channel_runs_pay


@pytest.mark.parametrize("lens,heads,d,dv,runs", [
    ([79], 16, 128, 128, False), ([80], 16, 128, 128, True), ([2047], 16, 128, 128, True), ([300], 1, 16, 16, False), ([300], 1, 32, 16, True),
    ([8] * 64, 16, 128, 128, False), ([128] * 64, 16, 128, 128, False), ([1] * 63 + [600], 16, 128, 128, True),
    ([1] * 63 + [600], 32, 128, 128, False), ([1] * 63 + [600], 16, 64, 64, True), ([1] * 63 + [600], 4, 64, 64, True), ([100] * 16, 16, 128, 128, False),
    ([128] * 16, 16, 128, 128, True), ([100] * 32, 2, 32, 32, True), ([100] * 32, 4, 64, 64, False)])
def test_delta_rule_in_runs(lens, heads, d, dv, runs):
    assert channel_runs_pay(lens, heads, d, dv) == runs
