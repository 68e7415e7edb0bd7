"""Expert kernels of CTA pairs (many tokens per expert): the edges of their token tiles, K remainders and row remainders,
against the CPU checker."""
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


def with_native(case, cfg, seed):
    tensors = [list(t) for t in (case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)]
    for e in range(cfg.total_experts - cfg.native_fp8_resources, cfg.total_experts):
        for i, t in enumerate(synthetic.native_fp8_tensors(cfg, seed, e)):
            tensors[i][e] = t
    return tensors


# K remainders of either stage (128 columns: one block; 384: a lone whole block after a pair; 576 = 4.5, 320 = 2.5, 704 = 5.5,
# 448 = 3.5 blocks: a half block after whole pairs, and after a lone block), weight rows that end inside a row tile and after
# the first of two (384, 576, 704), scale blocks of 32 and 128, a native FP8 resource; the rows a tile may have in either stage
# (`widths`), whose experts start at any row and end at any row of a tile, so that the last tiles run with fewer columns (the
# always-selected resource of the second configuration has every token)
@pytest.mark.parametrize("name,shape,tokens,native,widths", [
    ("gpt-oss-20b", (576, 320, 8), 400, 0, (128, 128)), ("gpt-oss-20b", (704, 448, 4), 241, 0, (64, 64)),
    ("gpt-oss-20b", (384, 128, 16), 499, 0, (64, 64)), ("gpt-oss-20b", (128, 192, 4), 97, 0, (64, 64)),
    ("deepseek-v3", (512, 384, 16), 240, 0, (128, 64)), ("deepseek-v3", (640, 256, 16), 481, 1, (128, 128)),
    ("deepseek-v3", (384, 640, 16), 193, 1, (128, 64)),
    ("gpt-oss-20b", (704, 448, 16), 940, 0, (240, 240)), ("gpt-oss-20b", (576, 320, 16), 700, 0, (192, 192)),
    ("gpt-oss-20b", (1152, 704, 8), 470, 0, (240, 240)), ("gpt-oss-20b", (640, 512, 16), 770, 0, (240, 240)),
    ("deepseek-v3", (640, 384, 16), 420, 1, (240, 240)), ("deepseek-v3", (768, 512, 16), 330, 0, (192, 192)),
    ("deepseek-v3", (640, 384, 16), 330, 1, (192, 192))])
def test_layer_matches_the_checker(device, name, shape, tokens, native, widths):
    cfg = synthetic.replace(synthetic.small_variant(synthetic.CONFIGS[name], *shape), native_fp8_resources=native)
    assert tokens * cfg.total_k > 96 * cfg.total_experts  # what takes a call to these kernels
    case = synthetic.make_case(cfg, tokens, seed=17)
    tensors = with_native(case, cfg, 17)
    plan = MoePlan.for_config(device, cfg, tokens)
    assert (plan.debug_token_tile(0, tokens), plan.debug_token_tile(1, tokens)) == ((widths[0], True), (widths[1], True))
    plan.set_expert_path(2)
    bank = ExpertBank.upload(device, *tensors)
    out = device.create_resident_buffer(tokens * cfg.hidden * 2)
    plan.layer(tokens, bank, device.resident_buffer_from(case.hidden), out, router_weights=device.resident_buffer_from(case.router_w),
               router_bias=device.resident_buffer_from(case.router_bias) if case.router_bias is not None else None,
               bias=device.resident_buffer_from(case.select_bias) if case.select_bias is not None else None)
    logits = mo.linear_bf16(case.hidden, case.router_w, case.router_bias)
    everyone = np.arange(tokens)
    want = sampled.layer_on_sample(cfg, case.hidden, logits, case.select_bias, everyone, lambda e: [t[e] for t in tensors])
    assert_close(out.read(np.uint16).reshape(tokens, cfg.hidden), want["output"], f"{name} {shape} CTA pairs T{tokens}")
    assert plan.status() == 0
    plan.destroy()
    bank.destroy()


# one matrix: of few rows (64 tokens a tile, whole and ragged last tiles), and of rows that fill the pairs once or twice, where
# tiles of 192 and 240 tokens are taken: the widths, a token less, a token more, two whole tiles
@pytest.mark.parametrize("rows,cols,tokens,width", [
    (256, 256, 97, 64), (288, 448, 128, 64), (160, 576, 129, 64), (384, 704, 192, 64), (256, 128, 193, 64), (320, 192, 240, 64),
    (544, 320, 241, 64), (1152, 640, 300, 64),
    (9888, 128, 191, 192), (9888, 192, 192, 192), (9888, 128, 193, 240), (9856, 192, 239, 240), (9888, 320, 240, 240),
    (18912, 128, 300, 192), (18912, 128, 385, 240), (18912, 192, 433, 240), (18912, 192, 480, 240)])
def test_dense_linear_matches_the_checker(device, rows, cols, tokens, width):
    rng = np.random.default_rng(rows + cols + tokens)
    plan = MoePlan.for_config(device, synthetic.MoeConfig("pairs", 256, 256, 8, 2, act_block=32), 480)
    shape = MoePlan.for_config(device, synthetic.MoeConfig("linear", rows, cols, 1, 1, act_block=32), tokens)  # its down stage
    assert shape.debug_token_tile(1, tokens) == (width, True)
    shape.destroy()
    plan.set_expert_path(2)
    x = synthetic.f32_to_bf16(rng.standard_normal((tokens, cols)).astype(np.float32))
    w, s = rng.integers(0, 256, (rows, cols // 2), dtype=np.uint8), rng.integers(118, 128, (rows, cols // 32), dtype=np.uint8)
    out = device.create_resident_buffer(tokens * rows * 2)
    plan.dense_linear(tokens, device.resident_buffer_from(x), out, device.resident_buffer_from(w), device.resident_buffer_from(s), rows, cols)
    assert_close(out.read(np.uint16).reshape(tokens, rows), mo.dense_linear_mxfp4(x, w, s, 32, tier=1))
    assert plan.status() == 0
    plan.destroy()


@pytest.mark.parametrize("cta", [0, 1])
def test_a_wait_that_expires_is_reported(device, cta):
    """Copies that one CTA of a pair leaves out, the announcement of both CTAs' (0) or only its own (1): both wind down, the call
    reports it, the next call is whole."""
    cfg = synthetic.small_variant(synthetic.CONFIGS["gpt-oss-20b"], 576, 320, 8)
    tokens = 400
    case = synthetic.make_case(cfg, tokens, seed=18)
    plan = MoePlan.for_config(device, cfg, tokens)
    plan.set_expert_path(2)
    bank = ExpertBank.upload(device, case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)
    hidden, rw = device.resident_buffer_from(case.hidden), device.resident_buffer_from(case.router_w)
    out = device.create_resident_buffer(tokens * cfg.hidden * 2)
    plan.layer(tokens, bank, hidden, out, router_weights=rw)
    assert plan.status() == 0
    before = out.read(np.uint16).copy()
    plan.set_wait_limit(2_000_000)  # about a millisecond
    plan.debug_withhold_arrival(1 + cta)
    plan.layer(tokens, bank, hidden, out, router_weights=rw)
    device.synchronize(timeout_ns=20_000_000_000)
    assert plan.status() & 8
    plan.debug_withhold_arrival(False)
    plan.set_wait_limit(0)
    for _ in range(2):
        plan.layer(tokens, bank, hidden, out, router_weights=rw)
        assert plan.status() == 0
        np.testing.assert_array_equal(out.read(np.uint16), before)
    plan.destroy()
    bank.destroy()


# K of one stage and of several, weight rows of one tile and of more, scale blocks of 32 and of 128 (the warps of a group hand
# maxima round in the middle of the exchange)
@pytest.mark.parametrize("name,shape,tokens", [("gpt-oss-20b", (128, 192, 4), 97), ("gpt-oss-20b", (704, 448, 4), 241), ("deepseek-v3", (512, 384, 16), 240)])
def test_waits_that_run_out_anywhere_leave_the_plan_whole(device, name, shape, tokens):
    cfg = synthetic.small_variant(synthetic.CONFIGS[name], *shape)
    case = synthetic.make_case(cfg, tokens, seed=33)
    plan = MoePlan.for_config(device, cfg, tokens)
    plan.set_expert_path(2)
    bank = ExpertBank.upload(device, case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)
    hidden, rw = device.resident_buffer_from(case.hidden), device.resident_buffer_from(case.router_w)
    bias = device.resident_buffer_from(case.select_bias) if case.select_bias is not None else None
    out = device.create_resident_buffer(tokens * cfg.hidden * 2)
    plan.layer(tokens, bank, hidden, out, router_weights=rw, bias=bias)
    assert plan.status() == 0
    before, seen = out.read(np.uint16).copy(), 0
    for limit in (1, 400, 1500, 4000, 20000):
        plan.set_wait_limit(limit)
        for _ in range(4):
            plan.layer(tokens, bank, hidden, out, router_weights=rw, bias=bias)
        device.synchronize(timeout_ns=20_000_000_000)
        seen |= plan.status()
    assert seen & ~8 == 0
    plan.set_wait_limit(0)
    plan.layer(tokens, bank, hidden, out, router_weights=rw, bias=bias)
    assert plan.status() == 0
    np.testing.assert_array_equal(out.read(np.uint16), before)
    plan.destroy()
    bank.destroy()


@pytest.mark.parametrize("rows,cols,tokens", [(288, 448, 130), (160, 2112, 40)])
def test_outputs_off_the_word_grid(device, rows, cols, tokens):
    """Outputs that start at an odd multiple of two bytes, which a lane stores one row of a token at a time instead of two: the same bits, nothing beside them."""
    from nerve_b200.backend import ResidentBuffer

    rng = np.random.default_rng(rows)
    plan = MoePlan.for_config(device, synthetic.MoeConfig("odd", 256, 256, 8, 2, act_block=32), tokens)
    plan.set_expert_path(2)
    x = device.resident_buffer_from(synthetic.f32_to_bf16(rng.standard_normal((tokens, cols)).astype(np.float32)))
    w, s = (device.resident_buffer_from(rng.integers(lo, hi, (rows, n), dtype=np.uint8)) for lo, hi, n in ((0, 256, cols // 2), (118, 128, cols // 32)))
    even, odd = (device.resident_buffer_from(np.full(tokens * rows + 8, 0x7fc0, dtype=np.uint16)) for _ in range(2))
    inner = ResidentBuffer.wrap(device, odd.device_address() + 2, tokens * rows * 2)
    plan.dense_linear(tokens, x, even, w, s, rows, cols)
    plan.dense_linear(tokens, x, inner, w, s, rows, cols)
    assert plan.status() == 0
    got, want = odd.read(np.uint16), even.read(np.uint16)
    np.testing.assert_array_equal(got[1:tokens * rows + 1], want[:tokens * rows])
    assert got[0] == 0x7fc0 and (got[tokens * rows + 1:] == 0x7fc0).all()
    plan.destroy()


def test_expert_rows_off_the_word_grid(device):
    """The same for a layer call whose expert rows the caller gets."""
    from nerve_b200.backend import ResidentBuffer

    cfg, tokens = synthetic.small_variant(synthetic.CONFIGS["gpt-oss-20b"], 576, 320, 8), 400
    case = synthetic.make_case(cfg, tokens, seed=17)
    plan = MoePlan.for_config(device, cfg, tokens)
    bank = ExpertBank.upload(device, case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)
    hidden, weights, bias = (device.resident_buffer_from(a) for a in (case.hidden, case.router_w, case.router_bias))
    count = tokens * cfg.total_k * cfg.hidden
    even, odd = (device.resident_buffer_from(np.full(count + 8, 0x7fc0, dtype=np.uint16)) for _ in range(2))
    for rows in (even, ResidentBuffer.wrap(device, odd.device_address() + 2, count * 2)):
        plan.layer(tokens, bank, hidden, None, router_weights=weights, router_bias=bias, expert_outputs=rows)
    assert plan.status() == 0
    got, want = odd.read(np.uint16), even.read(np.uint16)
    np.testing.assert_array_equal(got[1:count + 1], want[:count])
    assert got[0] == 0x7fc0 and (got[count + 1:] == 0x7fc0).all()
    plan.destroy()
    bank.destroy()


@pytest.mark.parametrize("shape,tokens", [((960, 2752, 96), 14216), ((1216, 1920, 128), 8868), ((768, 768, 64), 12000)])
def test_passes_agree(device, shape, tokens):
    """Short K, where the CTAs of a pair wait for each other's chunks: a chunk that is overwritten before it was read shows as rows that differ from pass to pass."""
    cfg = synthetic.small_variant(synthetic.CONFIGS["deepseek-v3"], *shape)
    cfg = synthetic.replace(cfg, act_block=128 if shape[0] % 128 == 0 and shape[1] % 128 == 0 else 32)
    rng = np.random.default_rng(shape[0])
    (H, I), E = shape[:2], cfg.total_experts
    mats = [m for r, c in ((I, H), (I, H), (H, I)) for m in (rng.integers(0, 256, (r, c // 2), dtype=np.uint8), rng.integers(118, 122, (r, c // 32), dtype=np.uint8))]
    bank = ExpertBank.upload(device, *([m] * E for m in mats))
    plan = MoePlan.for_config(device, cfg, tokens)
    buffer = device.resident_buffer_from
    hidden, weights = (buffer(synthetic.f32_to_bf16(rng.standard_normal(s, dtype=np.float32) * np.float32(f))) for s, f in (((tokens, H), 1), ((cfg.experts, H), 0.02)))
    bias = buffer(rng.standard_normal(cfg.experts, dtype=np.float32) * np.float32(0.05))
    out = device.create_resident_buffer(tokens * H * 2)
    first = None
    for _ in range(12):
        plan.layer(tokens, bank, hidden, out, router_weights=weights, bias=bias)
        got = out.read(np.uint16).reshape(tokens, H)
        first = got.copy() if first is None else first
        assert (got != first).any(axis=1).sum() == 0  # (rows)
    assert plan.status() == 0
    plan.destroy()
    bank.destroy()
