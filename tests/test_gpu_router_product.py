"""The bound that the router of large layer calls rests on: its tensor-core product lies within `relative` |x| |w| of the projection's sums (64 chains of
f32 additions, folded), for inputs that bring both near what they can err by, over every number of parts that the columns are split into. The share of the
bound that the product by itself, against 64-bit sums, may take is checked apart: it is what was measured of the tensor core's additions (16 units of
2^-24 a step of 16 columns where 10.5 are derived), and a device whose additions cut off earlier fails here."""
import numpy as np
import pytest

from nerve_b200 import synthetic
from nerve_b200.backend import CudaComputeDevice, MoePlan

pytestmark = pytest.mark.gpu

UNIT = 2.0 ** -24
TOKENS, EXPERTS = 130, 24  # (a whole tile of tokens and two rows; 24 is no multiple of 16)


@pytest.fixture(scope="module")
def device():
    dev = CudaComputeDevice(0)
    yield dev
    dev.close()


def pinned_sums(x, w):
    """The projection's sums in its own order, in f32 (a product of two bf16 numbers is exact in it)."""
    steps = x.shape[1] // 2 // 64
    acc = np.zeros((len(x), len(w), 64), dtype=np.float32)
    xs, ws = x.reshape(len(x), -1, 2), w.reshape(len(w), -1, 2)
    for s in range(steps + (x.shape[1] // 2 % 64 != 0)):
        lanes = min(64, x.shape[1] // 2 - 64 * s)
        for half in range(2):
            a, b = xs[:, 64 * s:64 * s + lanes, half], ws[:, 64 * s:64 * s + lanes, half]
            acc[:, :, :lanes] += a[:, None, :] * b[None, :, :]
    for fold in (32, 16, 8, 4, 2, 1):
        acc = acc + acc[:, :, np.arange(64) ^ fold]
    return acc[:, :, 0]


def rows(kind, hidden, rng):
    """Token and router rows as f32 values of bf16."""
    x, w = rng.standard_normal((TOKENS, hidden)), rng.standard_normal((EXPERTS, hidden)) * 0.02
    column = np.arange(hidden)
    if kind == "positive, the largest first":  # of every 16, 128 columns and of the row
        x, w = np.abs(x) + 0.5, np.abs(w) + 0.01
        x[:, column % 16 == 0] *= 1.9
        x[:, column % 128 == 0] *= 8
        x[:, 0] *= 64
    elif kind == "just below what is cut off":  # addends whose last bits lie under those of the first of their 16
        x, w = np.ones_like(x), np.ones_like(w)
        x[:, 1:] = rng.choice([2.0 ** -12, 2.0 ** -13], (TOKENS, hidden - 1)) * (1 + rng.integers(0, 128, (TOKENS, hidden - 1)) / 128)
        w[:, 1:] = rng.choice([2.0 ** -11, 2.0 ** -12], (EXPERTS, hidden - 1)) * (1 + rng.integers(0, 128, (EXPERTS, hidden - 1)) / 128)
        x[:, column % 16 == 0], w[:, column % 16 == 0] = 1.0, 1.0
    elif kind == "one step":  # all of the row in 16 columns
        x[:, 16:] = 0
        x = np.abs(x)
        w = np.abs(w)
    elif kind == "one flush":  # ... in 128
        x[:, 128:] = 0
        x, w = np.abs(x) + 0.25, np.abs(w) + 0.005
        x[:, 0] *= 16
    elif kind == "cancellation":
        x[:, 1::2] = -x[:, ::2] * (1 + rng.integers(-1, 2, (TOKENS, hidden // 2)) / 128)
        w[:, 1::2] = w[:, ::2]
    elif kind == "all magnitudes":
        x *= np.exp2(rng.integers(-12, 13, x.shape))
        w *= np.exp2(rng.integers(-12, 13, w.shape))
    elif kind == "outliers":
        x[:, rng.integers(0, hidden, 3)] *= 500
    bf16 = synthetic.f32_to_bf16
    return bf16(x.astype(np.float32)), bf16(w.astype(np.float32))


KINDS = ["normal", "positive, the largest first", "just below what is cut off", "one step", "one flush", "cancellation", "all magnitudes", "outliers"]


# one column block, one part; 2 to 8 parts; the longest rows in use
@pytest.mark.parametrize("hidden,parts", [(64, 1), (192, 1), (512, 2), (768, 3), (1024, 4), (1344, 5), (1536, 6), (1792, 7), (2048, 8), (2880, 8), (7168, 8)])
def test_product_lies_within_the_bound(device, hidden, parts):
    plan = MoePlan.for_config(device, synthetic.MoeConfig("p", hidden, 128, EXPERTS, 4, router_kind=synthetic.ROUTER_TOPK_SOFTMAX, act_block=32), TOKENS)
    most, apart = 0.0, 0.0
    for kind in KINDS:
        xb, wb = rows(kind, hidden, np.random.default_rng(hidden + len(kind)))
        product, x_norm, w_norm, relative, splits = plan.debug_router_product(TOKENS, device.resident_buffer_from(xb), device.resident_buffer_from(wb), EXPERTS)
        assert plan.status() == 0 and splits == parts
        x, w = synthetic.bf16_to_f32(xb), synthetic.bf16_to_f32(wb)
        x64, w64 = x.astype(np.float64), w.astype(np.float64)
        # (the norms are f32 sums of squares: a hundredth is far more than these err by)
        np.testing.assert_allclose(x_norm, np.linalg.norm(x64, axis=1), rtol=1e-2)
        np.testing.assert_allclose(w_norm, np.linalg.norm(w64, axis=1), rtol=1e-2)
        scale = x_norm[:, None].astype(np.float64) * w_norm
        ratio = np.abs(product.astype(np.float64) - pinned_sums(x, w)) / (relative * scale)
        assert ratio.max() <= 1.0, (kind, ratio.max())
        # eight steps a flush, an addition a flush, the parts
        units = 8 * 16 + hidden / 128 + 1 + splits
        alone = np.abs(product - x64 @ w64.T) / (units * UNIT * scale)
        assert alone.max() <= 1.0, (kind, alone.max())
        most, apart = max(most, ratio.max()), max(apart, alone.max())
    print(f"hidden {hidden}: {most:.3f} of the bound, {apart:.3f} of the product's share")
    plan.destroy()


def test_one_step_stays_within_what_is_derived(device):
    """A single step of 16 columns errs by no more than 10.5 units of the norms' product: 17 addends cut off 2^-25 below the largest, and the sum cut to 24 bits."""
    hidden = 64
    plan = MoePlan.for_config(device, synthetic.MoeConfig("p", hidden, 128, EXPERTS, 4, router_kind=synthetic.ROUTER_TOPK_SOFTMAX, act_block=32), TOKENS)
    for kind in KINDS:
        xb, wb = rows(kind, hidden, np.random.default_rng(len(kind)))
        xb[:, 16:] = 0
        product, x_norm, w_norm, _, _ = plan.debug_router_product(TOKENS, device.resident_buffer_from(xb), device.resident_buffer_from(wb), EXPERTS)
        x, w = synthetic.bf16_to_f32(xb).astype(np.float64), synthetic.bf16_to_f32(wb).astype(np.float64)
        # (the addends, not the rows, are what the largest is of: sum |x w| is at most |x| |w|)
        error = np.abs(product - x @ w.T) / (np.abs(x) @ np.abs(w).T)
        assert error.max() <= 10.5 * UNIT, (kind, error.max() / UNIT)
    plan.destroy()
