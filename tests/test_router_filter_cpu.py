"""What the filter of large layer calls relies on: the sigmoid of the router is monotone over all bf16 logits."""
import numpy as np

from oracle import moe_oracle as mo


def test_sigmoid_is_monotone_over_bf16():
    mo.build()
    expf = mo.lib().oracle_expf
    codes = np.concatenate([np.arange(0xff80, 0x7fff, -1), np.arange(0x0000, 0x7f81)]).astype(np.uint32)  # -inf .. -0, 0 .. inf
    values = (codes << 16).view(np.float32)
    one = np.float32(1)
    exps = np.array([expf(float(-v)) for v in values], dtype=np.float32)
    sigmoid = one / (one + exps)
    assert np.all(sigmoid[1:] >= sigmoid[:-1]) and sigmoid[0] == 0 and sigmoid[-1] == 1
