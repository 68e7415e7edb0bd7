"""Scheduling of layers with so many experts that a sort in one block is at the end of its shared memory: the largest count that the
one-block forms take, the next, and the counts at which their static arrays count beside the dynamic ones."""
import numpy as np
import pytest

from nerve_b200 import synthetic
from nerve_b200.backend import CudaComputeDevice, MoePlan, address_table, geometry_from_config
from oracle import moe_oracle as mo
from tests.helpers import assert_close, expert_params

pytestmark = pytest.mark.gpu

H, I, K, SETS = 128, 128, 4, 3  # (three sets of weights: expert e has those of e % 3)


@pytest.fixture(scope="module")
def device():
    dev = CudaComputeDevice(0)
    yield dev
    dev.close()


class Layer:
    def __init__(self, device, experts, tokens):
        rng = np.random.default_rng(experts + tokens)
        self.cfg = synthetic.MoeConfig("limits", H, I, experts, K, act_block=32)
        self.tokens, self.plan = tokens, MoePlan(device, geometry_from_config(self.cfg, tokens))
        self.hidden = synthetic.f32_to_bf16(rng.standard_normal((tokens, H), dtype=np.float32))
        ids = np.stack([np.sort(rng.choice(experts, K, replace=False)) for _ in range(tokens)]).astype(np.uint32)
        ids[0, -1] = experts - 1
        self.routes = synthetic.f32_to_bf16(rng.random((tokens, K), dtype=np.float32)).astype(np.uint32) << 16 | ids
        per = [[m for r, c in ((I, H), (I, H), (H, I)) for m in (rng.integers(0, 256, (r, c // 2), dtype=np.uint8),
                                                                 rng.integers(121, 128, (r, c // 32), dtype=np.uint8))] for _ in range(SETS)]
        which = np.arange(experts, dtype=np.uint32)[:, None] % SETS
        self.host = [[m for s in per for m in s[:4]], (which * 4 + np.arange(4, dtype=np.uint32)).ravel(),
                     [m for s in per for m in s[4:]], (which * 2 + np.arange(2, dtype=np.uint32)).ravel()]
        self.gate_addresses = address_table(device, [device.resident_buffer_from(m) for m in self.host[0]])
        self.down_addresses = address_table(device, [device.resident_buffer_from(m) for m in self.host[2]])
        self.gate_up_slots, self.down_slots = (device.resident_buffer_from(self.host[i]) for i in (1, 3))
        self.gate_up_addresses = self.gate_addresses

    def nodes(self, device):
        """The scheduled expert outputs of the node operators: schedule words and rows."""
        plan, T = self.plan, self.tokens
        routes, hidden = device.resident_buffer_from(self.routes), device.resident_buffer_from(self.hidden)
        control = np.array([T, 0, 0, 0, 0, 0, 0], dtype=np.uint32)
        gc, dc = device.resident_buffer_from(control), device.resident_buffer_from(control)
        frames, out = device.create_resident_buffer(T * plan.frame_words * 4), device.create_resident_buffer(T * K * H * 2)
        plan.moe_route_compact(T, routes, frames, gc, self.gate_up_slots)
        plan.independent_sparse_moe_gate_up(T, hidden, routes, frames, self.gate_addresses, self.gate_up_slots, gc)
        plan.moe_route_count(T, routes, dc, self.down_slots)
        plan.independent_sparse_moe_down(T, frames, routes, out, self.down_addresses, self.down_slots, dc)
        return frames.read(np.uint32).reshape(T, plan.frame_words), out.read(np.uint16).reshape(T, K, H)


# 300 routes (a block of 1024) and 256 (a block of 256); with static arrays forgotten, 645 and 646 or 1751 to 1755 experts pass 48 KB
@pytest.mark.parametrize("tokens,experts", [(75, 642), (75, 643), (75, 644), (75, 645), (75, 646), (75, 647),
                                            (64, 1745), (64, 1746), (64, 1747), (64, 1751), (64, 1755), (64, 1756)])
def test_node_operators_at_the_end_of_shared_memory(device, tokens, experts):
    case = Layer(device, experts, tokens)
    frames, got = case.nodes(device)
    ep = expert_params(case.cfg)
    want_frames, want = np.zeros_like(frames), np.zeros_like(got)
    control = np.array([tokens, 0, 0, 0, 0, 0, 0], dtype=np.uint32)
    mo.route_compact(case.routes, want_frames, control, I, K, 4, slots=case.host[1])
    np.testing.assert_array_equal(frames[:, case.plan.data_words:], want_frames[:, case.plan.data_words:])
    mo.gate_up(ep, case.hidden, case.routes, want_frames, mo.address_table(case.host[0]), case.host[1], control)
    mo.down(ep, want_frames, case.routes, want, mo.address_table(case.host[2]), case.host[3], np.array([tokens, 0, 0, 0, 0, 0, 0], dtype=np.uint32))
    assert_close(got.reshape(tokens * K, H), want.reshape(tokens * K, H), f"{experts} experts T{tokens} nodes")
    assert case.plan.status() == 0
    case.plan.destroy()


# 4096 routes, which the layer call sorts in one block while that has room
@pytest.mark.parametrize("experts", [2686, 2687, 2706, 2729, 2730])
def test_layer_call_at_the_end_of_shared_memory(device, experts):
    case = Layer(device, experts, 1024)
    _, want = case.nodes(device)
    got = device.create_resident_buffer(want.nbytes)
    case.plan.layer(case.tokens, case, device.resident_buffer_from(case.hidden), None, routes_in=device.resident_buffer_from(case.routes),
                    expert_outputs=got)
    np.testing.assert_array_equal(got.read(np.uint16).reshape(want.shape), want)
    assert case.plan.status() == 0
    case.plan.destroy()
