"""Layer calls of at most 1024 routes of all experts, whose operands are made beside the schedule: edges of the block sizes (a route a
thread of 256, 512 or 1024), of 32 experts and of 512 columns, one token and 1024 routes, experts that a stage lacks, tokens that cannot be
routed, routes and logits of the caller's. A call that is profiled schedules first and quantises then: the same bits."""
import numpy as np
import pytest

from nerve_b200 import synthetic
from nerve_b200.backend import CudaComputeDevice, ExpertBank, MoePlan

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device():
    dev = CudaComputeDevice(0)
    yield dev
    dev.close()


class Layer:
    def __init__(self, device, name, shape, tokens, **changes):
        self.cfg = cfg = synthetic.replace(synthetic.small_variant(synthetic.CONFIGS[name], *shape), **changes)
        self.case = case = synthetic.make_case(cfg, tokens, seed=7)
        self.device, self.tokens, self.plan = device, tokens, MoePlan.for_config(device, cfg, tokens)
        self.bank = ExpertBank.upload(device, case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)
        buffer = lambda a: None if a is None else device.resident_buffer_from(a)
        self.hidden = buffer(case.hidden)
        self.args = dict(router_weights=buffer(case.router_w), router_bias=buffer(case.router_bias), bias=buffer(case.select_bias))
        self.out = device.create_resident_buffer(tokens * cfg.hidden * 2)
        self.routes = device.create_resident_buffer(tokens * cfg.total_k * 4)

    def call(self, profiled, **args):
        """Output, routes, telemetry and status of a call."""
        self.plan.set_profiling(profiled)
        telemetry = self.device.resident_buffer_from(np.zeros(self.plan.telemetry_words(), dtype=np.uint32))
        if "routes_in" not in args:
            args = dict(args, routes_out=self.routes, telemetry=telemetry)
        self.out.write_bytes(np.full(self.tokens * self.cfg.hidden, 0x7fc0, dtype=np.uint16))
        self.plan.layer(self.tokens, self.bank, self.hidden, self.out, **args)
        got = [self.out.read(np.uint16).copy(), telemetry.read(np.uint32).copy()]
        if "routes_in" not in args:
            got.append(self.routes.read(np.uint32).copy())
        return got, self.plan.status()

    def same_both_ways(self, **args):
        args = args or self.args
        self.call(False, **args)  # (builds the tables of the experts)
        (got, status), (want, want_status) = self.call(False, **args), self.call(True, **args)
        assert status == want_status
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)
        return status

    def close(self):
        self.plan.destroy()
        self.bank.destroy()


# four routes a token (gpt-oss), nine with the shared expert (deepseek); hidden below, at and above one and two pieces of 512 columns
@pytest.mark.parametrize("name,shape,tokens", [
    ("tiny", (128, 128, 4), 1), ("gpt-oss-20b", (512, 128, 31), 8), ("gpt-oss-20b", (544, 128, 32), 9), ("gpt-oss-20b", (1024, 192, 32), 17),
    ("gpt-oss-20b", (1088, 128, 32), 32), ("gpt-oss-20b", (256, 128, 32), 33), ("gpt-oss-20b", (320, 128, 33), 16), ("gpt-oss-20b", (320, 128, 33), 17),
    ("gpt-oss-20b", (320, 128, 128), 15), ("gpt-oss-20b", (512, 128, 65), 64), ("gpt-oss-20b", (512, 128, 65), 65), ("gpt-oss-20b", (128, 128, 16), 255),
    ("gpt-oss-20b", (576, 128, 40), 256), ("gpt-oss-20b", (576, 128, 40), 257), ("deepseek-v3", (512, 128, 64), 1), ("deepseek-v3", (640, 256, 256), 29),
    ("deepseek-v3", (1152, 128, 48), 113), ("deepseek-v3", (384, 128, 256), 114)])
def test_operands_beside_the_schedule(device, name, shape, tokens):
    layer = Layer(device, name, shape, tokens)
    assert layer.same_both_ways() == 0
    layer.close()


# the projection by wide tiles from 444 of them on, which a profiled call takes from 740 on: 440, 448 and 512 of them
@pytest.mark.parametrize("name,shape,tokens", [("gpt-oss-20b", (1088, 128, 64), 220), ("gpt-oss-20b", (1088, 128, 64), 224), ("gpt-oss-20b", (576, 128, 127), 127)])
def test_projection_by_wide_tiles_beside_operands(device, name, shape, tokens):
    test_operands_beside_the_schedule(device, name, shape, tokens)


# many routes a token: either side of the lines from which on the schedule comes first (routed in the same blocks, by eight warps, by 32)
@pytest.mark.parametrize("k,hidden,tokens", [
    (16, 1088, 8), (16, 512, 8), (32, 2048, 4), (32, 1024, 4), (32, 512, 16), (12, 1024, 21), (12, 512, 21), (6, 1088, 170), (6, 512, 170), (16, 2880, 30), (16, 2880, 64),
    (32, 512, 32)])
def test_many_routes_a_token(device, k, hidden, tokens):
    layer = Layer(device, "gpt-oss-20b", (hidden, 128, 64), tokens, k=k)
    assert layer.same_both_ways() == 0
    layer.close()


# ... which lie further out where there are many experts: routed ahead of the blocks, and in them
@pytest.mark.parametrize("k,hidden,tokens,experts", [
    (12, 512, 49, 192), (12, 960, 38, 192), (24, 704, 4, 256), (24, 320, 12, 256), (16, 320, 64, 256), (7, 320, 45, 8), (20, 1472, 7, 128), (31, 320, 8, 128), (7, 320, 27, 9), (31, 320, 2, 48)])
def test_many_routes_of_many_experts(device, k, hidden, tokens, experts):
    layer = Layer(device, "gpt-oss-20b", (hidden, 128, experts), tokens, k=k)
    assert layer.same_both_ways() == 0
    layer.close()


@pytest.mark.parametrize("tokens", [5, 20, 200])
def test_experts_that_a_stage_lacks(device, tokens):
    layer = Layer(device, "gpt-oss-20b", (1088, 192, 32), tokens)
    selected = [int(w) & 0xffff for w in layer.call(False, **layer.args)[0][2][:4]]
    unbound = np.full(4, 0xffffffff, dtype=np.uint32)
    for e in selected[:2]:
        layer.bank.gate_up_slots.write_bytes(unbound, offset=4 * 4 * e)
    for e in selected[1:3]:
        layer.bank.down_slots.write_bytes(unbound[:2], offset=2 * 4 * e)
    assert layer.same_both_ways() != 0
    layer.close()


@pytest.mark.parametrize("tokens", [3, 31, 100])
def test_tokens_that_cannot_be_routed_and_callers_logits(device, tokens):
    layer = Layer(device, "gpt-oss-20b", (576, 128, 32), tokens)
    rng = np.random.default_rng(tokens)
    logits = synthetic.f32_to_bf16(rng.standard_normal((tokens, 32), dtype=np.float32))
    logits[0] = 0x3f80  # (equal scores)
    assert layer.same_both_ways(logits=device.resident_buffer_from(logits)) == 0
    logits[tokens // 2] = 0x7fc0  # NaN: no selectable score
    assert layer.same_both_ways(logits=device.resident_buffer_from(logits)) != 0
    layer.close()


@pytest.mark.parametrize("shape,tokens", [((576, 128, 32), 2), ((2048, 1280, 32), 60), ((320, 128, 40), 256)])
def test_routes_of_the_caller(device, shape, tokens):
    """Among them some of no expert (the second shape's call takes one launch for both expert stages)."""
    layer = Layer(device, "gpt-oss-20b", shape, tokens)
    rng = np.random.default_rng(tokens)
    ids = np.stack([np.sort(rng.choice(shape[2], 4, replace=False)) for _ in range(tokens)]).astype(np.uint32)
    for bad in (False, True):
        if bad:
            ids[1::3, 3] = 0xffff
            ids[0, 2] = shape[2]
        routes = synthetic.f32_to_bf16(rng.random((tokens, 4), dtype=np.float32)).astype(np.uint32) << 16 | ids
        assert (layer.same_both_ways(routes_in=device.resident_buffer_from(routes)) != 0) == bad
    layer.close()


def test_successive_calls_of_other_tokens(device):
    """Rows that are read before the wait are those of this call: four inputs in turn, without a pause, on one plan."""
    layer = Layer(device, "gpt-oss-20b", (2880, 192, 32), 24)
    rng = np.random.default_rng(1)
    sources = [device.resident_buffer_from(synthetic.f32_to_bf16(rng.standard_normal((24, 2880), dtype=np.float32) * np.float32(s))) for s in (1, 50, 1e-3, 7)]
    want = []
    for layer.hidden in sources:
        want.append(layer.call(True, **layer.args)[0])
    outs = [device.create_resident_buffer(24 * 2880 * 2) for _ in range(16)]
    layer.plan.set_profiling(False)
    copies, zeros = device.create_resident_buffer(24 * 2880 * 2), device.resident_buffer_from(np.zeros((24, 2880), dtype=np.uint16))
    layer.plan.layer(24, layer.bank, sources[0], outs[0], **layer.args)
    for n, out in enumerate(outs):
        # the tokens come from an operator of this library that lets the next start early
        layer.plan.residual_add(24, 2880, sources[n % 4], zeros, copies)
        layer.plan.layer(24, layer.bank, copies, out, **layer.args)
    for n, out in enumerate(outs):
        np.testing.assert_array_equal(out.read(np.uint16), want[n % 4][0])
    layer.close()
