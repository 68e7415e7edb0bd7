"""silu_multiply over all 65536 bf16 gates, bounded and not, against the pinned form: whatever the hardware's exponential settles has the same bits."""
import numpy as np
import pytest

from nerve_b200 import synthetic
from nerve_b200.backend import CudaComputeDevice, MoePlan
from oracle import moe_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [0.0, 7.0, 100.0, 3e38])
def test_all_gates(limit):
    device = CudaComputeDevice(0)
    rng = np.random.default_rng(int(limit))
    ups = synthetic.f32_to_bf16((rng.standard_normal(48) * np.exp(rng.uniform(-20, 20, 48))).astype(np.float32))
    ups = np.concatenate([ups, np.array([0x3f80, 0xbf80, 0x0000, 0x8000, 0x7f80, 0xff80, 0x7fc0, 0x0001, 0x7f7f, 0x3f81, 0x40e0, 0xc0e1, 0x0080, 0x4f00, 0x3001, 0xbfff],
                                         dtype=np.uint16)])
    gates = np.tile(np.arange(65536, dtype=np.uint32).astype(np.uint16), (len(ups), 1))
    u = np.repeat(ups[:, None], 65536, axis=1)
    u[0] = synthetic.f32_to_bf16(rng.standard_normal(65536).astype(np.float32))  # (a row with another u each)
    plan = MoePlan.for_config(device, synthetic.MoeConfig("silu", 256, 256, 8, 2, act_block=32), len(ups))
    out = device.create_resident_buffer(gates.nbytes)
    plan.silu_multiply(len(ups), 65536, device.resident_buffer_from(gates), device.resident_buffer_from(u), out, limit)
    g, up = synthetic.bf16_to_f32(gates), synthetic.bf16_to_f32(u)
    numbers = ~np.isnan(g) & ~np.isnan(up)
    with np.errstate(all="ignore"):
        if limit:
            g, up = np.fmin(g, np.float32(limit)), np.fmin(np.fmax(up, np.float32(-limit)), np.float32(limit))
        # (which NaN a NaN is, the host and the device settle differently; an infinite factor makes one of any act that rounds to zero)
        number = numbers & ~np.isnan(g / (1 + np.exp(-g)) * up) & ~(np.isinf(up) & (np.abs(g / (1 + np.exp(-g))) < 1e-30))
    got, want = out.read(np.uint16).reshape(gates.shape), mo.silu_multiply(gates, u, limit)
    np.testing.assert_array_equal(got[number], want[number])
    plan.destroy()
    device.close()


@pytest.mark.parametrize("limit", [6.9999, 7.1, 0.3, 88.7])
def test_bounds_that_are_no_bf16_number(limit):
    """The bounded gate is then any f32 number."""
    test_all_gates(limit)


@pytest.mark.parametrize("limit", [0.0, 7.0])
def test_zeros(limit):
    """Zeros of either sign by gates and ups of either, small, large and below the exponential's range: the zero that the pinned form makes."""
    device = CudaComputeDevice(0)
    zeros, others = np.array([0x0000, 0x8000]), np.array([0x0000, 0x8000, 0x3f80, 0xbf80, 0x0080, 0x8001, 0x4120, 0xc120, 0xc2ae, 0xc2b0, 0xc2b2, 0xc2b4, 0xc2c8, 0x7f7f, 0xff7f, 0x7f00])
    pairs = [(z, o) for z in zeros for o in others] + [(o, z) for z in zeros for o in others]
    gates, ups = (np.tile(np.array([p[i] for p in pairs], dtype=np.uint16), (3, 8)) for i in (0, 1))
    plan = MoePlan.for_config(device, synthetic.MoeConfig("silu", 256, 256, 8, 2, act_block=32), 3)
    out = device.create_resident_buffer(gates.nbytes)
    plan.silu_multiply(3, gates.shape[1], device.resident_buffer_from(gates), device.resident_buffer_from(ups), out, limit)
    np.testing.assert_array_equal(out.read(np.uint16).reshape(gates.shape), mo.silu_multiply(gates, ups, limit))
    plan.destroy()
    device.close()


def test_fast_activation_errs_by_less_than_its_check_allows():
    """Over every gate that there can be: positive f32 numbers (the bound can be any) and negative bf16 numbers."""
    device = CudaComputeDevice(0)
    units, allowed = device.debug_silu_units()
    print(f"{units} units of {allowed}")
    assert 0 < units <= allowed
    device.close()
