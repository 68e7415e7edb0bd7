"""Layer calls on host buffers: page-locked rows that kernels read and write, rows off the 16-byte grid, at the end of an allocation
and beyond the size for it, pageable rows; the results are those of the call on resident buffers."""
import numpy as np
import pytest

from nerve_b200 import synthetic
from nerve_b200.backend import CudaComputeDevice, ExpertBank, MoePlan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [1, 33, 9000])  # (9000 rows of 512 columns: 9.2 MB, by copies)
def test_host_rows(tokens):
    torch = pytest.importorskip("torch")
    device = CudaComputeDevice(0)
    cfg = synthetic.small_variant(synthetic.CONFIGS["gpt-oss-20b"], 512, 128, 8)
    case = synthetic.make_case(cfg, tokens, seed=47)
    plan = MoePlan.for_config(device, cfg, tokens)
    bank = ExpertBank.upload(device, case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)
    rw = device.resident_buffer_from(case.router_w)
    out = device.create_resident_buffer(tokens * cfg.hidden * 2)
    plan.layer(tokens, bank, device.resident_buffer_from(case.hidden), out, router_weights=rw)
    want = out.read(np.uint16).reshape(tokens, cfg.hidden)
    count = tokens * cfg.hidden

    def rows(pinned, offset):  # the last `count` words of an allocation that is `offset` words longer
        if not pinned:
            return np.zeros(count + offset, dtype=np.uint16)[offset:].reshape(tokens, cfg.hidden)
        return torch.zeros(count + offset, dtype=torch.int16).pin_memory().numpy().view(np.uint16)[offset:].reshape(tokens, cfg.hidden)

    for pinned_in, offset_in, pinned_out, offset_out in ((True, 0, True, 0), (True, 8, True, 24), (True, 3, True, 0), (True, 0, True, 1),
                                                         (False, 0, True, 0), (True, 0, False, 0), (False, 1, False, 1)):
        x, y = rows(pinned_in, offset_in), rows(pinned_out, offset_out)
        x[...] = case.hidden
        plan.layer_host(tokens, bank, x, y, router_weights=rw)
        np.testing.assert_array_equal(y, want)
    x, y = rows(True, 0), rows(True, 0)
    x[...] = case.hidden
    plan.layer_host(tokens, bank, x, x, router_weights=rw)  # in place
    np.testing.assert_array_equal(x, want)
    assert plan.status() == 0
    plan.destroy()
    bank.destroy()
    device.close()


@pytest.mark.parametrize("words", [0, 8, 5])  # of an offset on the 16-byte grid and off it
def test_registered_host_rows(words):
    """Pageable memory that the caller has registered counts as page-locked."""
    torch = pytest.importorskip("torch")
    device = CudaComputeDevice(0)
    tokens = 21
    cfg = synthetic.small_variant(synthetic.CONFIGS["gpt-oss-20b"], 512, 128, 8)
    case = synthetic.make_case(cfg, tokens, seed=47)
    plan = MoePlan.for_config(device, cfg, tokens)
    bank = ExpertBank.upload(device, case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)
    rw = device.resident_buffer_from(case.router_w)
    out = device.create_resident_buffer(tokens * cfg.hidden * 2)
    plan.layer(tokens, bank, device.resident_buffer_from(case.hidden), out, router_weights=rw)
    whole = np.zeros(2 * 4096 + 2 * tokens * cfg.hidden, dtype=np.uint16)  # (whole pages inside it are registered)
    start = -(-whole.ctypes.data // 4096) * 4096
    size = (whole.ctypes.data + whole.nbytes - start) // 4096 * 4096
    assert int(torch.cuda.cudart().cudaHostRegister(start, size, 0)) == 0
    first = (start - whole.ctypes.data) // 2 + words
    count = tokens * cfg.hidden
    x, y = (whole[first + i * count:first + (i + 1) * count].reshape(tokens, cfg.hidden) for i in (0, 1))
    assert y.ctypes.data + y.nbytes <= start + size
    x[...] = case.hidden
    for _ in range(2):
        y[...] = 0
        plan.layer_host(tokens, bank, x, y, router_weights=rw)
        np.testing.assert_array_equal(y, out.read(np.uint16).reshape(tokens, cfg.hidden))
    assert int(torch.cuda.cudart().cudaHostUnregister(start)) == 0
    plan.destroy()
    bank.destroy()
    device.close()
