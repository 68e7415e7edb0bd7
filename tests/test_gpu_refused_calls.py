"""A layer call that is refused launches nothing and leaves what the plan reports of the last whole call."""
import numpy as np
import pytest

from nerve_b200 import synthetic
from nerve_b200.backend import CudaComputeDevice, CudaError, ExpertBank, MoePlan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("profiled", [False, True])
def test_refused_layer_calls(profiled):
    device = CudaComputeDevice(0)
    tokens = 9
    cfg = synthetic.small_variant(synthetic.CONFIGS["deepseek-v3"], 256, 128, 16)
    case = synthetic.make_case(cfg, tokens, seed=53)
    plan = MoePlan.for_config(device, cfg, tokens)
    plan.set_profiling(profiled)
    bank = ExpertBank.upload(device, case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)
    hidden, out = device.resident_buffer_from(case.hidden), device.create_resident_buffer(tokens * cfg.hidden * 2)
    good = {"router_weights": device.resident_buffer_from(case.router_w), "bias": device.resident_buffer_from(case.select_bias)}
    plan.layer(tokens, bank, hidden, out, **good)
    small = device.create_resident_buffer(4)
    before, launches = plan.last_report(), plan.launches()
    assert before["total_ms"] > 0.0
    x, y = case.hidden.copy(), np.zeros_like(case.hidden)
    for bad in ({"telemetry": small}, {"bias": small}, {"bias": None}, {"logits": small}, {"router_weights": small}, {"router_bias": small},
                {"routes_out": small}):
        with pytest.raises(CudaError):
            plan.layer(tokens, bank, hidden, out, **(good | bad))
        with pytest.raises(CudaError):
            plan.layer_host(tokens, bank, x, y, **(good | bad))
        assert plan.launches() == launches, bad
        assert plan.last_report() == before, bad
    assert not y.any()
    plan.layer_host(tokens, bank, x, y, **good)
    np.testing.assert_array_equal(y, out.read(np.uint16).reshape(y.shape))
    assert plan.launches() > launches and plan.status() == 0
    plan.destroy()
    bank.destroy()
    device.close()


def test_profiling_turned_on_after_the_call():
    """A report asked for with profiling on, after a call without it, has no stage times and leaves no error behind."""
    device = CudaComputeDevice(0)
    tokens = 9
    cfg = synthetic.small_variant(synthetic.CONFIGS["gpt-oss-20b"], 256, 128, 16)
    case = synthetic.make_case(cfg, tokens, seed=59)
    plan = MoePlan.for_config(device, cfg, tokens)
    bank = ExpertBank.upload(device, case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)
    hidden, out = device.resident_buffer_from(case.hidden), device.create_resident_buffer(tokens * cfg.hidden * 2)
    rw = device.resident_buffer_from(case.router_w)
    for profiled, asked in ((False, True), (True, True), (True, False), (False, True), (False, False)):
        plan.set_profiling(profiled)
        plan.layer(tokens, bank, hidden, out, router_weights=rw)
        plan.set_profiling(asked)
        report = plan.last_report()
        times = [*report["stage_ms"].values(), report["gate_up_kernel_ms"], report["down_kernel_ms"]]
        assert any(times) == (profiled and asked) and report["total_ms"] > 0.0
    assert plan.status() == 0
    plan.destroy()
    bank.destroy()
    device.close()
