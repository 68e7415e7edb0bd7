"""Both expert stages of a layer call in one launch (calls of more than a round of gate/up tiles): token tiles of every width, K
and row remainders, one-byte weight forms, experts that only one stage holds, waits that run out, against the CPU checker."""
import numpy as np
import pytest

from nerve_b200 import synthetic
from nerve_b200.backend import CudaComputeDevice, ExpertBank, MoePlan
from oracle import moe_oracle as mo
from oracle import sampled
from tests.helpers import assert_close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device():
    dev = CudaComputeDevice(0)
    yield dev
    dev.close()


def prepared(device, name, shape, tokens, native=0):
    cfg = synthetic.replace(synthetic.small_variant(synthetic.CONFIGS[name], *shape), native_fp8_resources=native)
    case = synthetic.make_case(cfg, tokens, seed=41)
    tensors = [list(t) for t in (case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)]
    for e in range(cfg.total_experts - native, cfg.total_experts):
        for i, t in enumerate(synthetic.native_fp8_tensors(cfg, 41, e)):
            tensors[i][e] = t
    plan = MoePlan.for_config(device, cfg, tokens)
    bank = ExpertBank.upload(device, *tensors)
    out = device.create_resident_buffer(tokens * cfg.hidden * 2)
    hidden, rw = device.resident_buffer_from(case.hidden), device.resident_buffer_from(case.router_w)
    kw = dict(router_weights=rw, router_bias=device.resident_buffer_from(case.router_bias) if case.router_bias is not None else None,
              bias=device.resident_buffer_from(case.select_bias) if case.select_bias is not None else None)
    return cfg, case, tensors, plan, bank, out, lambda: plan.layer(tokens, bank, hidden, out, **kw)


# 32 or 33 experts x 5 to 7 row tiles of gate/up; K of 2.5, 5.5, 1.5 and whole blocks; down rows that end in the first or the second
# half of a tile; tokens an expert for tiles of 16, 32, 64 and 96
@pytest.mark.parametrize("name,shape,tokens,native", [
    ("gpt-oss-20b", (320, 704, 32), 40, 0), ("gpt-oss-20b", (192, 832, 32), 130, 0), ("gpt-oss-20b", (576, 640, 32), 290, 0),
    ("gpt-oss-20b", (320, 704, 32), 700, 0), ("gpt-oss-20b", (128, 640, 32), 33, 0),
    ("deepseek-v3", (384, 640, 32), 35, 1), ("deepseek-v3", (256, 768, 32), 75, 1), ("deepseek-v3", (640, 640, 32), 340, 1)])
def test_layer_matches_the_checker(device, name, shape, tokens, native):
    cfg, case, tensors, plan, bank, out, call = prepared(device, name, shape, tokens, native)
    for _ in range(2):  # (the second call finds the counters of the first)
        call()
        assert plan.status() == 0
        logits = mo.linear_bf16(case.hidden, case.router_w, case.router_bias)
        want = sampled.layer_on_sample(cfg, case.hidden, logits, case.select_bias, np.arange(tokens), lambda e: [t[e] for t in tensors])
        assert_close(out.read(np.uint16).reshape(tokens, cfg.hidden), want["output"], f"{name} {shape} one launch T{tokens}")
    # projection, router, schedule (three launches from 1280 routes on), quantisation, both expert stages, combine
    assert plan.last_report()["kernel_launches"] == (6 if tokens * cfg.total_k < 1280 else 8)
    plan.destroy()
    bank.destroy()


@pytest.mark.parametrize("name,shape,tokens,native", [
    ("gpt-oss-20b", (1920, 1152, 32), 40, 0), ("gpt-oss-20b", (2624, 1216, 32), 160, 0), ("gpt-oss-20b", (2752, 1088, 32), 290, 0),
    ("gpt-oss-20b", (3008, 1152, 32), 700, 0), ("deepseek-v3", (2048, 1280, 32), 35, 1), ("deepseek-v3", (3072, 1280, 32), 340, 0)])
def test_successive_calls_hand_over_their_own_rows(device, name, shape, tokens, native):
    """Calls of the same plan on tokens of very different size: a down tile that read codes or scales from before its gate/up tiles
    were done would find those of the call ahead. The outputs are those of launches of their own (a profiled call)."""
    cfg, case, tensors, plan, bank, out, call = prepared(device, name, shape, tokens, native)
    rng = np.random.default_rng(3)
    rw = device.resident_buffer_from(case.router_w)
    kw = dict(router_weights=rw, router_bias=device.resident_buffer_from(case.router_bias) if case.router_bias is not None else None,
              bias=device.resident_buffer_from(case.select_bias) if case.select_bias is not None else None)
    sources = [device.resident_buffer_from(synthetic.f32_to_bf16(rng.standard_normal((tokens, cfg.hidden), dtype=np.float32) * np.float32(size)))
               for size in (1.0, 1e-3, 60.0)]
    want = []
    plan.set_profiling(True)
    for source in sources:
        plan.layer(tokens, bank, source, out, **kw)
        want.append(out.read(np.uint16).copy())
    plan.set_profiling(False)
    for i in (0, 1, 2, 1, 0, 2, 0, 1, 1, 2):
        plan.layer(tokens, bank, sources[i], out, **kw)
        np.testing.assert_array_equal(out.read(np.uint16), want[i])
    assert plan.last_report()["kernel_launches"] == (6 if tokens * cfg.total_k < 1280 else 8)  # (one launch for both stages)
    assert plan.status() == 0
    plan.destroy()
    bank.destroy()


# Either side of the lines of the rule: K of gate/up by token tile (16, 32, 64, 96), K of down, rounds of gate/up, tiles of down
@pytest.mark.parametrize("shape,tokens,one", [
    ((1408, 1152, 32), 64, False), ((1536, 1152, 32), 64, True), ((2304, 1152, 32), 160, False), ((2432, 1152, 32), 160, True),
    ((2432, 1152, 32), 290, False), ((2560, 1152, 32), 290, True), ((2816, 1152, 32), 700, False), ((2944, 1152, 32), 700, True),
    ((2048, 896, 40), 40, False), ((2048, 960, 40), 40, True), ((3968, 384, 80), 720, False), ((4096, 384, 80), 720, True),
    ((512, 896, 32), 40, True), ((512, 960, 32), 40, False), ((1792, 1536, 32), 5, False), ((1792, 1536, 32), 6, True)])
def test_which_calls_take_one_launch(device, shape, tokens, one):
    cfg, case, tensors, plan, bank, out, call = prepared(device, "gpt-oss-20b", shape, tokens)
    got = []
    call()  # (builds the tables of the experts)
    for profiled in (False, True):
        plan.set_profiling(profiled)
        call()
        got.append(out.read(np.uint16).copy())
        if not profiled:  # projection, router, schedule, quantisation, one or two, combine; up to 32 tokens route in the schedule
            separate = 8 if tokens * cfg.total_k >= 1280 else 6 if tokens > 32 else 5
            assert plan.last_report()["kernel_launches"] == separate + (0 if one else 1)
    np.testing.assert_array_equal(got[0], got[1])
    assert plan.status() == 0
    plan.destroy()
    bank.destroy()


def test_experts_that_one_stage_lacks(device):
    """An expert without down weights, one without gate/up weights (whose down rows are zeros) and one without either: the same
    output as from the launches of their own that a profiled call makes."""
    cfg, case, tensors, plan, bank, out, call = prepared(device, "gpt-oss-20b", (320, 704, 32), 96)
    unbound = np.full(4, 0xffffffff, dtype=np.uint32)
    gate, down = bank.gate_up_slots, bank.down_slots
    down.write_bytes(unbound[:2], offset=2 * 4 * 3)
    gate.write_bytes(unbound, offset=4 * 4 * 5)
    gate.write_bytes(unbound, offset=4 * 4 * 31)
    down.write_bytes(unbound[:2], offset=2 * 4 * 31)
    got = []
    for profiled in (False, True):
        plan.set_profiling(profiled)
        call()
        assert plan.status() != 0  # (experts that are not resident)
        got.append(out.read(np.uint16).copy())
    np.testing.assert_array_equal(got[0], got[1])
    plan.destroy()
    bank.destroy()


@pytest.mark.parametrize("tokens", [20, 200, 500])
def test_expert_ranges(device, tokens):
    """Calls of a range of the experts: the same output as from launches of their own, and routes of other experts count as zeros."""
    cfg, case, tensors, plan, bank, out, call = prepared(device, "gpt-oss-20b", (320, 704, 32), tokens)
    hidden, rw = device.resident_buffer_from(case.hidden), device.resident_buffer_from(case.router_w)
    rbias = device.resident_buffer_from(case.router_bias)
    for start, count in ((0, 32), (0, 9), (9, 23), (31, 1)):
        got = []
        for profiled in (False, True, False):
            plan.set_profiling(profiled)
            plan.layer(tokens, bank, hidden, out, router_weights=rw, router_bias=rbias, expert_start=start, expert_count=count)
            assert plan.status() == 0
            got.append(out.read(np.uint16).copy())
        np.testing.assert_array_equal(got[0], got[1])
        np.testing.assert_array_equal(got[0], got[2])
        assert 0.0 < plan.last_report()["total_ms"] < 1000.0
    plan.destroy()
    bank.destroy()


@pytest.mark.parametrize("name,shape,tokens", [("gpt-oss-20b", (320, 704, 32), 40), ("gpt-oss-20b", (1152, 640, 32), 700), ("deepseek-v3", (384, 640, 32), 35)])
def test_waits_that_run_out_anywhere_leave_the_plan_whole(device, name, shape, tokens):
    cfg, case, tensors, plan, bank, out, call = prepared(device, name, shape, tokens)
    call()
    assert plan.status() == 0
    before, seen = out.read(np.uint16).copy(), 0
    for limit in (1, 400, 1500, 4000, 20000):
        plan.set_wait_limit(limit)
        for _ in range(4):
            call()
        device.synchronize(timeout_ns=20_000_000_000)
        seen |= plan.status()
    assert seen & ~8 == 0
    plan.set_wait_limit(2_000_000)  # about a millisecond
    plan.debug_withhold_arrival(True)
    call()
    device.synchronize(timeout_ns=20_000_000_000)
    assert plan.status() & 8
    plan.debug_withhold_arrival(False)
    plan.set_wait_limit(0)
    for _ in range(2):
        call()
        assert plan.status() == 0
        np.testing.assert_array_equal(out.read(np.uint16), before)
    plan.destroy()
    bank.destroy()
