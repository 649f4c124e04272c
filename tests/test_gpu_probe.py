"""The rate probes that the benchmark divides by: within what the pipes can do."""
import pytest
import torch

import ves

pytestmark = pytest.mark.gpu


def test_rates_within_issue_limits():
    props = torch.cuda.get_device_properties(0)
    per_clk = props.multi_processor_count * 2.07e9
    fp64, fp32, imad = (f() / per_clk for f in (ves.fp64_fma_rate, ves.fp32_fma_rate, ves.imad_wide_rate))
    assert 1.5 < fp64 / 2 < 2.1 and 64 < fp32 / 2 <= 128
    assert 16 < imad <= 64  # a 64-bit result takes two register writes: at most half the FP32 rate
    again = ves.imad_wide_rate() / per_clk
    assert abs(again - imad) <= 0.05 * imad
