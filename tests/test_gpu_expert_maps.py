"""Calls of more experts than a block acquires tensor maps of before its first copy (both stages in one launch): the last number of experts that it does, the first beyond, more than
threads of the acquiring warp take in one pass, one-byte weights among them, K short enough that a block's tiles follow one another at once. The bytes are
those of launches of their own (a profiled call)."""
import numpy as np
import pytest

from tests.test_gpu_layer_launch import device, prepared  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,shape,tokens,native", [
    ("gpt-oss-20b", (320, 384, 64), 40, 0), ("gpt-oss-20b", (320, 384, 65), 40, 0), ("gpt-oss-20b", (128, 256, 110), 90, 0), ("gpt-oss-20b", (640, 128, 200), 80, 0),
    ("gpt-oss-20b", (2048, 960, 100), 60, 0), ("deepseek-v3", (384, 384, 64), 35, 1)])
def test_many_experts_in_one_launch(device, name, shape, tokens, native):  # noqa: F811
    cfg, case, tensors, plan, bank, out, call = prepared(device, name, shape, tokens, native)
    plan.set_profiling(True)
    call()
    want = out.read(np.uint16).copy()
    plan.set_profiling(False)
    for _ in range(3):
        out.fill(0xFF)
        call()
        assert plan.status() == 0
        np.testing.assert_array_equal(out.read(np.uint16), want)
    assert plan.last_report()["kernel_launches"] == 6  # one for both stages
    plan.destroy()
    bank.destroy()


# ... acquired tile by tile (short K, or few tiles a block) and, with long K and many, beside the first copies; one-byte weights among either
@pytest.mark.parametrize("name,shape,tokens,native", [
    ("gpt-oss-20b", (2176, 1152, 100), 60, 0), ("gpt-oss-20b", (2176, 1088, 90), 60, 0), ("deepseek-v3", (2304, 1280, 128), 40, 1), ("deepseek-v3", (1536, 1024, 128), 30, 1),
    ("gpt-oss-20b", (1536, 1024, 200), 100, 0)])
def test_maps_by_tile_and_beside(device, name, shape, tokens, native):  # noqa: F811
    test_many_experts_in_one_launch(device, name, shape, tokens, native)
