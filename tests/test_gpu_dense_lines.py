"""Dense linears of few tokens: either side of the lines from which on they run by CTA pairs (25 tokens with 2048 columns and more, 49 with
fewer), with whole and ragged last tiles of 64 tokens, K and row remainders, and calls of fewer tokens on a plan of more, against the oracle."""
import numpy as np
import pytest

from nerve_b200 import synthetic
from nerve_b200.backend import CudaComputeDevice, MoePlan
from oracle import moe_oracle as mo
from tests.helpers import assert_close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device():
    dev = CudaComputeDevice(0)
    yield dev
    dev.close()


@pytest.mark.parametrize("rows,cols,most,calls", [
    (288, 2048, 25, (25, 24, 12, 1)), (160, 2112, 48, (33, 48, 25)), (544, 2240, 64, (64, 49, 24)), (256, 2304, 96, (96, 65, 26, 5)),
    (288, 1984, 48, (48, 25)), (160, 576, 49, (49, 48)), (384, 1920, 96, (96, 64, 49)), (96, 2176, 97, (97, 96, 25)), (320, 704, 200, (200, 70, 30))])
def test_dense_linear_of_few_tokens(device, rows, cols, most, calls):
    rng = np.random.default_rng(rows + cols)
    plan = MoePlan.for_config(device, synthetic.MoeConfig("lines", 256, 256, 8, 2, act_block=32), most)
    plan.set_expert_path(2)
    w, s = rng.integers(0, 256, (rows, cols // 2), dtype=np.uint8), rng.integers(118, 128, (rows, cols // 32), dtype=np.uint8)
    wb, sb = device.resident_buffer_from(w), device.resident_buffer_from(s)
    for tokens in calls:
        x = synthetic.f32_to_bf16(rng.standard_normal((tokens, cols)).astype(np.float32))
        out = device.create_resident_buffer(tokens * rows * 2)
        plan.dense_linear(tokens, device.resident_buffer_from(x), out, wb, sb, rows, cols)
        assert_close(out.read(np.uint16).reshape(tokens, rows), mo.dense_linear_mxfp4(x, w, s, 32, tier=1))
        assert plan.status() == 0
    plan.destroy()


def test_a_wait_that_expires_is_reported(device):
    rng = np.random.default_rng(1)
    rows, cols, tokens = 384, 2048, 40
    plan = MoePlan.for_config(device, synthetic.MoeConfig("lines", 256, 256, 8, 2, act_block=32), tokens)
    plan.set_expert_path(2)
    x = synthetic.f32_to_bf16(rng.standard_normal((tokens, cols)).astype(np.float32))
    w, s = rng.integers(0, 256, (rows, cols // 2), dtype=np.uint8), rng.integers(118, 128, (rows, cols // 32), dtype=np.uint8)
    args = (device.resident_buffer_from(x), device.create_resident_buffer(tokens * rows * 2), device.resident_buffer_from(w), device.resident_buffer_from(s))
    plan.set_wait_limit(2_000_000)  # about a millisecond
    plan.debug_withhold_arrival(True)
    plan.dense_linear(tokens, *args, rows, cols)
    device.synchronize(timeout_ns=20_000_000_000)
    assert plan.status() & 8
    plan.debug_withhold_arrival(False)
    plan.set_wait_limit(0)
    plan.dense_linear(tokens, *args, rows, cols)
    assert plan.status() == 0
    assert_close(args[1].read(np.uint16).reshape(tokens, rows), mo.dense_linear_mxfp4(x, w, s, 32, tier=1))
    plan.destroy()
