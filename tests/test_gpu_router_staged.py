"""The router projection of small calls with its rows staged in shared memory, against the oracle: the same bits on both sides of each line of its rule (blocks of one token by
two outputs, of two by four, the loads through registers in small and wide tiles), with odd tokens and outputs, rows that fill no whole step and the longest staged rows."""
import numpy as np
import pytest

from nerve_b200 import synthetic
from nerve_b200.backend import CudaComputeDevice, MoePlan, geometry_from_config
from oracle import moe_oracle as mo

pytestmark = pytest.mark.gpu

ONE_BY_TWO = [(1, 256, 2), (1, 2880, 33), (3, 544, 31), (128, 288, 4), (1, 8192, 31), (2, 96, 255)]
TWO_BY_FOUR = [(5, 1536, 131), (8, 1536, 295), (3, 8192, 255), (65, 2880, 33)]
THROUGH_REGISTERS = [(129, 288, 4), (9, 1504, 131), (9, 1536, 259), (2, 8224, 9)]
WIDE = [(221, 320, 63), (147, 1088, 192), (223, 288, 127), (245, 320, 113)]  # tiles of 4 x 8: 888 blocks with eight steps, 896 and 930 with four; 448 are too few by themselves


@pytest.mark.parametrize("tokens,hidden,outputs", ONE_BY_TWO + TWO_BY_FOUR + THROUGH_REGISTERS + WIDE)
def test_staged_projection_is_bit_exact(tokens, hidden, outputs):
    rng = np.random.default_rng(tokens * 1000 + outputs)
    x = synthetic.f32_to_bf16(rng.standard_normal((tokens, hidden), dtype=np.float32))
    w = synthetic.f32_to_bf16(0.02 * rng.standard_normal((outputs, hidden), dtype=np.float32))
    bias = synthetic.f32_to_bf16(0.1 * rng.standard_normal(outputs).astype(np.float32)) if outputs % 2 else None
    x[-1, -5:] = 0x8000  # negative zeros at a row's end
    want = mo.linear_bf16(x, w, bias)
    device = CudaComputeDevice(0)
    config = synthetic.MoeConfig(name="t", experts=outputs, k=1, hidden=hidden, intermediate=128, act_block=32)
    plan = MoePlan(device, geometry_from_config(config, tokens))
    guard = np.full(want.nbytes + 64, 0xA5, np.uint8)
    logits = device.resident_buffer_from(guard)
    plan.linear(tokens, device.resident_buffer_from(x), logits, device.resident_buffer_from(w), device.resident_buffer_from(bias) if bias is not None else None)
    np.testing.assert_array_equal(logits.read(np.uint32, want.size).reshape(want.shape), want)
    assert (logits.read(np.uint8, 64, want.nbytes) == 0xA5).all()  # nothing behind the last row
    plan.destroy()
    device.close()


# small tiles on either side of the line at 740 wide ones, 754 and 735 (with operands beside the line is lower: test_gpu_small_calls.py)
@pytest.mark.parametrize("tokens,hidden,outputs", [(229, 320, 101), (196, 576, 120)])
def test_line_of_the_wide_tiles(tokens, hidden, outputs):
    test_staged_projection_is_bit_exact(tokens, hidden, outputs)
