"""dequant_swiglu_quant on rows of odd length: one wave holds as many rows as the SMs do."""
import pytest
import torch

from helpers import best_time

pytestmark = pytest.mark.gpu


def test_eight_rows_per_sm_are_one_wave(ops):
    """A third more rows than six per SM: 1.25 times the time, 1.9 when eight blocks of the 32-register form are counted
    as six and the rest waits for a second wave."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    few, many = (torch.randn(n * sms, 2 * 3001, device="cuda").half() for n in (6, 8))
    t_few = best_time(lambda: ops.dequant_swiglu_quant(few, None, None, None, True))
    t_many = best_time(lambda: ops.dequant_swiglu_quant(many, None, None, None, True))
    assert t_many < 1.55 * t_few
