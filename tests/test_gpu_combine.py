"""The combine over 16-byte pieces against its definition (an f32 sum rounded to bf16 after every add, as whole-number arithmetic on the
bits): every kind of value, NaN, infinities, subnormals and halfway cases among them, route counts around the steps of four and nine."""
import numpy as np
import pytest

from nerve_b200 import synthetic
from nerve_b200.backend import CudaComputeDevice, ExpertBank, MoePlan, ResidentBuffer, geometry_from_config
from oracle import moe_oracle as mo

pytestmark = pytest.mark.gpu


def as_f32(halves):
    return (halves.astype(np.uint32) << 16).view(np.float32)


def rounded(values):
    """The bits of f32 values as bf16; a NaN the arithmetic makes has all mantissa bits set, and its rounding carries into the sign."""
    bits = np.where(np.isnan(values), np.uint32(0x7fffffff), values.astype(np.float32).view(np.uint32)).astype(np.uint64)
    return ((bits + 0x7fff + ((bits >> 16) & 1)) >> 16 & 0xffff).astype(np.uint16)


def combined(rows, scale):
    acc = np.zeros(rows.shape[::2], dtype=np.uint16)
    with np.errstate(all="ignore"):
        for r in range(rows.shape[1]):
            acc = rounded(as_f32(acc) + as_f32(rows[:, r]))
        return rounded(as_f32(acc) * np.float32(scale))


@pytest.mark.parametrize("k", [1, 3, 4, 5, 8, 9, 10])
@pytest.mark.parametrize("values", ["any bits", "near each other", "drawn"])
def test_combine_matches_its_definition(k, values):
    device = CudaComputeDevice(0)
    cfg = synthetic.replace(synthetic.small_variant(synthetic.CONFIGS["gpt-oss-20b"], 320, 64, 16), k=k)
    tokens, rng = 211, np.random.default_rng(k)
    geometry = geometry_from_config(cfg, tokens)
    geometry.reduce_scale = 2.5
    plan = MoePlan(device, geometry)
    shape = (tokens, cfg.total_k, cfg.hidden)
    if values == "any bits":  # one value in 128 is an infinity or a NaN
        rows = rng.integers(0, 1 << 16, shape, dtype=np.uint16)
    elif values == "near each other":  # sums that lie half-way, cancel, or leave the range
        rows = (rng.choice([0x0000, 0x0070, 0x3f80, 0x7f70], shape) + rng.integers(0, 16, shape) + 0x8000 * rng.integers(0, 2, shape)).astype(np.uint16)
    else:
        rows = rounded(rng.standard_normal(shape).astype(np.float32))
    source = device.resident_buffer_from(rows)
    out = device.create_resident_buffer(tokens * cfg.hidden * 2 + 16)
    want = combined(rows, 2.5)
    plan.moe_reduce(tokens, source, out)
    np.testing.assert_array_equal(out.read(np.uint16)[:want.size].reshape(want.shape), want)
    # the same from the kernel for rows that are not on the 16-byte grid
    shifted = ResidentBuffer.wrap(device, out.device_address() + 4, tokens * cfg.hidden * 2)
    plan.moe_reduce(tokens, source, shifted)
    np.testing.assert_array_equal(out.read(np.uint16)[2:2 + want.size].reshape(want.shape), want)
    shifted.destroy()
    plan.destroy()
    device.close()


# as many blocks of 16-byte pieces as rows are fetched with their marks in (296, 148 of nine routes), and one more (after them)
@pytest.mark.parametrize("name,tokens", [("gpt-oss-20b", 1894), ("gpt-oss-20b", 1895), ("deepseek-v3", 947), ("deepseek-v3", 948)])
def test_combine_leaves_skipped_routes_out(name, tokens):
    """Routes of an expert that is not resident and of experts out of a call's range count as zeros, whatever an earlier call left in
    their rows."""
    device = CudaComputeDevice(0)
    cfg = synthetic.replace(synthetic.small_variant(synthetic.CONFIGS[name], 320, 128, 16), act_block=32)
    case = synthetic.make_case(cfg, tokens, seed=61)
    plan = MoePlan.for_config(device, cfg, tokens)
    bank = ExpertBank.upload(device, case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)
    hidden, rw = device.resident_buffer_from(case.hidden), device.resident_buffer_from(case.router_w)
    kw = dict(router_weights=rw, router_bias=device.resident_buffer_from(case.router_bias) if case.router_bias is not None else None,
              bias=device.resident_buffer_from(case.select_bias) if case.select_bias is not None else None)
    out, rows = device.create_resident_buffer(tokens * cfg.hidden * 2), device.create_resident_buffer(tokens * cfg.total_k * cfg.hidden * 2)
    scale = geometry_from_config(cfg, tokens).reduce_scale
    loud = device.resident_buffer_from(np.full_like(case.hidden, 0x7f00))  # (finite, sums of which are not)
    bank.down_slots.write_bytes(np.full(2, 0xffffffff, dtype=np.uint32), offset=8 * 3)
    for start, count in ((0, 0), (0, 7), (5, cfg.total_experts - 5)):
        plan.layer(tokens, bank, loud, out, **kw)
        plan.layer(tokens, bank, hidden, out, expert_start=start, expert_count=count, **kw)
        got = out.read(np.uint16).reshape(tokens, cfg.hidden)
        plan.layer(tokens, bank, hidden, None, expert_start=start, expert_count=count, expert_outputs=rows, **kw)
        np.testing.assert_array_equal(got, mo.reduce(rows.read(np.uint16).reshape(tokens, cfg.total_k, cfg.hidden), tokens, cfg.total_k, cfg.hidden, scale))
    plan.destroy()
    bank.destroy()
    device.close()
