"""Large layer calls, whose logits are only made exactly where they matter: experts, weights, telemetry and output of a call that hands all its exact
logits to the caller (the pinned projection and the router on them), word for word. Edges of the token tile, of 64 and 128 columns, of 16, 32 and
128 experts; group-limited routing; and inputs for which the matrix product says little: ties, cancellation, zeros, NaN, infinities, the ends of
the range."""
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
        self.device, self.tokens, self.plan = device, tokens, MoePlan.for_config(device, cfg, tokens)
        rng = np.random.default_rng(5)
        tensors = [[None] * cfg.total_experts for _ in range(6)]
        H, I = cfg.hidden, cfg.intermediate
        shared = [m for r, c in ((I, H), (I, H), (H, I)) for m in (rng.integers(0, 256, (r, c // 2), dtype=np.uint8), rng.integers(118, 122, (r, c // 32), dtype=np.uint8))]
        for e in range(cfg.total_experts):
            for i in range(6):
                tensors[i][e] = shared[i]
        self.bank = ExpertBank.upload(device, *tensors)
        bf16 = synthetic.f32_to_bf16
        self.w = bf16(rng.standard_normal((cfg.experts, H), dtype=np.float32) * np.float32(0.02))
        self.x = bf16(rng.standard_normal((tokens, H), dtype=np.float32))
        self.logit_bias = bf16(rng.standard_normal(cfg.experts, dtype=np.float32) * np.float32(0.1)) if cfg.logit_bias else None
        self.select_bias = (rng.standard_normal(cfg.experts, dtype=np.float32) * np.float32(0.05)) if cfg.bias_dtype == synthetic.BIAS_F32 else None

    def both_ways(self):
        """Routes, telemetry, output and status with the filter, and with logits that the caller gets."""
        buffer = lambda a: None if a is None else self.device.resident_buffer_from(a)
        cfg, T = self.cfg, self.tokens
        hidden = buffer(self.x)
        logits = self.device.create_resident_buffer(T * ((cfg.experts + 1) // 2) * 4)
        args = dict(router_weights=buffer(self.w), router_bias=buffer(self.logit_bias), bias=buffer(self.select_bias))
        results = []
        for extra in ({}, {"logits": logits}):
            routes, telemetry = buffer(np.full((T, cfg.total_k), 0xdeadbeef, dtype=np.uint32)), buffer(np.zeros(self.plan.telemetry_words(), dtype=np.uint32))
            out = buffer(np.full((T, cfg.hidden), 0x7fc0, dtype=np.uint16))
            self.plan.layer(T, self.bank, hidden, out, routes_out=routes, telemetry=telemetry, **args, **extra)
            results.append((routes.read(np.uint32).copy(), telemetry.read(np.uint32).copy(), out.read(np.uint16).copy(), self.plan.status()))
        for got, want in zip(*results):
            np.testing.assert_array_equal(got, want)
        return results[0]

    def close(self):
        self.plan.destroy()
        self.bank.destroy()


# (which of them the rule of router_filter_takes filters: test_which_projection_a_call_uses)
@pytest.mark.parametrize("name,shape,tokens,changes", [
    ("gpt-oss-20b", (1152, 64, 16), 300, {}), ("gpt-oss-20b", (2880, 64, 128), 592, {}), ("gpt-oss-20b", (2880, 64, 32), 256, {}),
    ("gpt-oss-20b", (1408, 128, 16), 257, {}), ("gpt-oss-20b", (1472, 128, 17), 385, {}), ("gpt-oss-20b", (1152, 64, 5), 511, {}),
    ("gpt-oss-20b", (1792, 128, 32), 513, {}), ("gpt-oss-20b", (2880, 64, 33), 1100, {}), ("gpt-oss-20b", (2112, 64, 128), 2051, {}),
    ("gpt-oss-20b", (4096, 64, 129), 600, {}), ("gpt-oss-20b", (3584, 64, 256), 640, {"k": 8}), ("deepseek-v3", (7168, 128, 256), 1024, {}),
    ("deepseek-v3", (2560, 128, 64), 1300, {}), ("deepseek-v3", (2432, 128, 256), 601, {"n_group": 0, "topk_group": 0}),
    ("deepseek-v3", (2432, 128, 256), 767, {"n_group": 32, "topk_group": 5}), ("deepseek-v3", (1920, 128, 32), 1029, {"n_group": 32, "topk_group": 9}),
    ("deepseek-v3", (1536, 128, 16), 1100, {"n_group": 4, "topk_group": 1, "k": 4}), ("deepseek-v3", (1664, 128, 24), 1027, {"n_group": 0, "topk_group": 0, "k": 8}),
    ("gpt-oss-20b", (1024, 64, 32), 19000, {})])
def test_what_is_selected(device, name, shape, tokens, changes):
    layer = Layer(device, name, shape, tokens, **changes)
    assert layer.both_ways()[3] == 0
    layer.close()


def inputs(kind, layer):
    rng = np.random.default_rng(11)
    bf16, f32 = synthetic.f32_to_bf16, synthetic.bf16_to_f32
    x, w = f32(layer.x).copy(), f32(layer.w).copy()
    T, H = x.shape
    if kind == "ties":  # experts in equal pairs and one of all zeros; tokens in equal pairs, some of all zeros
        w[1::2] = w[0:len(w) - len(w) % 2:2][: len(w[1::2])]
        w[len(w) // 2] = 0
        x[1::2] = x[0::2][: len(x[1::2])]
        x[5:70] = 0
        x[70:90] = -0.0
    elif kind == "all the same":
        w[:] = w[0]
    elif kind == "cancellation":  # |x| |w| is a thousand times what is left
        x += 40
        w -= w.mean(axis=1, keepdims=True)
    elif kind == "close experts":  # a few units of the last place between them
        w[:] = w[0]
        w *= 1 + rng.integers(-2, 3, w.shape) / 256
    elif kind == "heavy":
        x, w = x ** 5, w ** 3
    elif kind == "tiny":
        x, w = x * np.float32(1e-25), w * np.float32(1e-12)
    elif kind == "subnormal":
        x = x * np.float32(1e-38)
    elif kind == "huge":
        x = x * np.float32(1e18)
    elif kind == "overflow":
        x, w = x * np.float32(1e25), w * np.float32(1e14)
    elif kind == "token specials":
        x[3, 7], x[130, 0], x[131, 1], x[132, 2:4], x[1000, 60] = np.nan, np.inf, -np.inf, (np.inf, -np.inf), 3e38
    elif kind == "expert specials":
        w[1, 3], w[2, 0], w[5, 5], w[7] = np.nan, np.inf, -np.inf, 3e38
    layer.x, layer.w = bf16(x.astype(np.float32)), bf16(w.astype(np.float32))
    if kind == "token specials":
        layer.x[3, 7] = 0x7fc0
    if kind == "expert specials":
        layer.w[1, 3] = 0x7fc0
    if kind == "bias specials":
        if layer.logit_bias is not None:
            layer.logit_bias[[1, 2, 4]] = (0x7fc0, 0x7f80, 0xff80)
        if layer.select_bias is not None:
            layer.select_bias[[1, 2, 4]] = (np.nan, np.inf, -np.inf)


@pytest.mark.parametrize("name,shape,changes", [("gpt-oss-20b", (1856, 64, 32), {}), ("gpt-oss-20b", (1728, 64, 100), {"k": 6}), ("deepseek-v3", (2560, 128, 64), {})])
@pytest.mark.parametrize("kind", ["ties", "all the same", "cancellation", "close experts", "heavy", "tiny", "subnormal", "huge", "overflow", "token specials",
                                  "expert specials", "bias specials"])
def test_inputs_that_the_product_says_little_of(device, name, shape, changes, kind):
    layer = Layer(device, name, shape, 1050, **changes)
    inputs(kind, layer)
    layer.both_ways()
    layer.close()


def test_a_wait_that_runs_out(device):
    """The status says so, routes stay in range, and the next call is whole."""
    layer = Layer(device, "gpt-oss-20b", (2880, 64, 32), 1024)
    want = layer.both_ways()
    layer.plan.set_wait_limit(1)
    buffer = layer.device.resident_buffer_from
    args = dict(router_weights=buffer(layer.w), router_bias=buffer(layer.logit_bias))
    routes, out = buffer(np.zeros((1024, 4), dtype=np.uint32)), buffer(np.zeros((1024, 2880), dtype=np.uint16))
    for _ in range(4):
        layer.plan.layer(1024, layer.bank, buffer(layer.x), out, routes_out=routes, **args)
        device.synchronize(timeout_ns=20_000_000_000)
        assert layer.plan.status() & ~8 == 0
        assert (routes.read(np.uint32) & 0xffff).max() < 32
    layer.plan.set_wait_limit(0)
    got = layer.both_ways()
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
    layer.close()


# sizes that the rule leaves to the projection by itself: few columns in one round of its blocks, 256 tokens; groups in one round
BELOW = [((1152, 64, 16), 300), ((2880, 64, 32), 256), ((1920, 128, 32), 1029), ((1536, 128, 16), 1100), ((2560, 128, 64), 1050)]
SELECTED = [tuple(case) for case in test_what_is_selected.pytestmark[0].args[1]]
UNTOLD = [(name, shape, 1050, changes) for name, shape, changes in
          next(mark.args[1] for mark in test_inputs_that_the_product_says_little_of.pytestmark if mark.args[0] == "name,shape,changes")]


# groups in one round of blocks, on either side of its lines: 32 experts or fewer by their columns, up to 128 in a round nearly full; many experts without groups
ONE_ROUND = [("deepseek-v3", (3072, 128, 32), 1029, {"n_group": 32, "topk_group": 9}, True), ("deepseek-v3", (2944, 128, 32), 700, {}, False),
             ("deepseek-v3", (2688, 128, 16), 1100, {"n_group": 4, "topk_group": 1, "k": 4}, True), ("deepseek-v3", (2560, 128, 64), 1057, {}, True),
             ("deepseek-v3", (4096, 128, 128), 545, {}, True), ("deepseek-v3", (4096, 128, 128), 300, {}, False), ("deepseek-v3", (7168, 128, 256), 257, {}, False),
             ("gpt-oss-20b", (4864, 64, 160), 417, {}, True), ("gpt-oss-20b", (4864, 64, 160), 330, {}, False)]


@pytest.mark.parametrize("name,shape,tokens,changes,filtered", ONE_ROUND)
def test_one_round_of_blocks(device, name, shape, tokens, changes, filtered):
    test_what_is_selected(device, name, shape, tokens, changes)
    layer = Layer(device, name, shape, tokens, **changes)
    buffer = lambda a: None if a is None else device.resident_buffer_from(a)
    layer.plan.layer(tokens, layer.bank, buffer(layer.x), device.create_resident_buffer(tokens * layer.cfg.hidden * 2), router_weights=buffer(layer.w),
                     router_bias=buffer(layer.logit_bias), bias=buffer(layer.select_bias))
    assert layer.plan.debug_projection() == filtered and layer.plan.status() == 0
    layer.close()


@pytest.mark.parametrize("kind", [kind for mark in test_inputs_that_the_product_says_little_of.pytestmark if mark.args[0] == "kind" for kind in mark.args[1]])
def test_groups_by_a_product_that_says_little(device, kind):
    """The inputs above, of groups in a size that the filter takes."""
    layer = Layer(device, "deepseek-v3", (2560, 128, 64), 1057)
    inputs(kind, layer)
    layer.both_ways()
    layer.close()


@pytest.mark.parametrize("name,shape,tokens,changes", SELECTED + UNTOLD)
def test_which_projection_a_call_uses(device, name, shape, tokens, changes):
    """The calls that the tests above compare: with the filter unless the caller gets the logits, or they lie below its line."""
    layer = Layer(device, name, shape, tokens, **changes)
    buffer = lambda a: None if a is None else device.resident_buffer_from(a)
    hidden, out = buffer(layer.x), device.create_resident_buffer(tokens * layer.cfg.hidden * 2)
    logits = device.create_resident_buffer(tokens * ((layer.cfg.experts + 1) // 2) * 4)
    args = dict(router_weights=buffer(layer.w), router_bias=buffer(layer.logit_bias), bias=buffer(layer.select_bias))
    for extra in ({}, {"logits": logits}):
        layer.plan.layer(tokens, layer.bank, hidden, out, **args, **extra)
        assert layer.plan.debug_projection() == ((shape, tokens) not in BELOW and not extra)
    assert layer.plan.status() == 0
    layer.close()


@pytest.mark.parametrize("name,shape,tokens,changes", [*UNTOLD[:2], ("deepseek-v3", (2560, 128, 64), 1057, {})])
def test_rows_that_the_product_errs_most_by(device, name, shape, tokens, changes):
    """Positive ones, the largest first, by experts a step or two apart."""
    layer = Layer(device, name, shape, tokens, **changes)
    rng = np.random.default_rng(11)
    x, w = (np.abs(synthetic.bf16_to_f32(a)) for a in (layer.x, layer.w))
    x += 0.5
    x[:, ::128] *= 8
    x[:, 0] *= 64
    w[:] = w[0] + 0.01
    w *= 1 + rng.integers(-1, 2, w.shape) / 256
    layer.x, layer.w = synthetic.f32_to_bf16(x.astype(np.float32)), synthetic.f32_to_bf16(w.astype(np.float32))
    layer.both_ways()
    layer.close()


# (some clocks, about as many as the product takes, so that the roles give up at different places; every one that does holds its CTA two milliseconds)
@pytest.mark.parametrize("limit", [300, 1500, 5000])
def test_waits_that_may_run_out(device, limit):
    """Whichever of the waits run out: no status but theirs, routes in range, and the next call is whole."""
    layer = Layer(device, "gpt-oss-20b", (2880, 64, 32), 1024)
    want = layer.both_ways()
    layer.plan.set_wait_limit(limit)
    buffer = layer.device.resident_buffer_from
    args = dict(router_weights=buffer(layer.w), router_bias=buffer(layer.logit_bias))
    routes, out = buffer(np.zeros((1024, 4), dtype=np.uint32)), buffer(np.zeros((1024, 2880), dtype=np.uint16))
    for _ in range(4):
        layer.plan.layer(1024, layer.bank, buffer(layer.x), out, routes_out=routes, **args)
        device.synchronize(timeout_ns=20_000_000_000)
        assert layer.plan.status() & ~8 == 0
        assert (routes.read(np.uint32) & 0xffff).max() < 32
    layer.plan.set_wait_limit(0)
    for a, b in zip(layer.both_ways(), want):
        np.testing.assert_array_equal(a, b)
    layer.close()


@pytest.mark.parametrize("name,shape,tokens", [("gpt-oss-20b", (2880, 64, 32), 1024), ("gpt-oss-20b", (2880, 64, 128), 2051), ("deepseek-v3", (2560, 128, 64), 1300)])
def test_a_copy_that_does_not_come(device, name, shape, tokens):
    """The first CTA of the product waits for a stage that is left out: the status says so, routes are in range, the other CTAs' tokens are whole, and so is
    the next call."""
    layer = Layer(device, name, shape, tokens)
    want = layer.both_ways()
    layer.plan.set_wait_limit(2_000_000)  # about a millisecond
    layer.plan.debug_withhold_arrival(3)
    buffer = lambda a: None if a is None else device.resident_buffer_from(a)
    cfg = layer.cfg
    routes, out = buffer(np.zeros((tokens, cfg.total_k), dtype=np.uint32)), buffer(np.zeros((tokens, cfg.hidden), dtype=np.uint16))
    layer.plan.layer(tokens, layer.bank, buffer(layer.x), out, routes_out=routes, router_weights=buffer(layer.w), router_bias=buffer(layer.logit_bias),
                     bias=buffer(layer.select_bias))
    device.synchronize(timeout_ns=20_000_000_000)
    assert layer.plan.status() == 8
    got = routes.read(np.uint32)
    assert (got & 0xffff).max() < cfg.total_experts
    np.testing.assert_array_equal(got.reshape(tokens, -1)[128:], want[0].reshape(tokens, -1)[128:])
    layer.plan.debug_withhold_arrival(0)
    layer.plan.set_wait_limit(0)
    for a, b in zip(layer.both_ways(), want):
        np.testing.assert_array_equal(a, b)
    layer.close()


@pytest.mark.parametrize("shape,tokens,k,fits", [((1024, 128, 256), 2304, 8, True), ((3584, 64, 256), 2304, 2, True), ((1536, 64, 256), 1400, 1, False)])
def test_scratch_is_shared_with_the_expert_rows(device, shape, tokens, k, fits):
    """A plan's first layer call takes what its logits, routes, frames and expert rows need, and nothing for the product where that is no more than the rows."""
    import torch

    layer = Layer(device, "gpt-oss-20b", shape, tokens, k=k)
    buffer = device.resident_buffer_from
    args = dict(router_weights=buffer(layer.w), router_bias=buffer(layer.logit_bias))
    hidden, out = buffer(layer.x), buffer(np.zeros((tokens, shape[0]), dtype=np.uint16))
    device.synchronize()
    before = torch.cuda.mem_get_info(0)[0]
    layer.plan.layer(tokens, layer.bank, hidden, out, **args)
    device.synchronize()
    taken = before - torch.cuda.mem_get_info(0)[0]
    rows, product = tokens * k * shape[0] * 2, min(8 * tokens, 148 * 128) * (shape[2] + 1) * 4
    assert (product <= rows) == fits
    others = tokens * (shape[2] // 2 * 4 + k * 4 + layer.plan.frame_words * 4)
    scales = shape[2] * 3 * -(-shape[0] // 128) * -(-shape[1] // 128) * 512  # of the experts, in the kernels' order
    # (each allocation is rounded up to 2 MiB)
    assert taken <= max(rows, product) + others + scales + (8 << 20), (taken, rows, product, others, scales)
    layer.close()
