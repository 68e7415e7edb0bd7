"""Sizes at which the launch rules change kernels, and the remainders inside them: against the CPU checker, or (the layer
call and its nodes, rows off the 16-byte grid, routes without gate/up) against another form of the same work."""
import numpy as np
import pytest

from nerve_b200 import synthetic
from nerve_b200.backend import CudaComputeDevice, CudaError, ExpertBank, MoePlan, ResidentBuffer, geometry_from_config
from oracle import moe_oracle as mo
from oracle import sampled
from tests.helpers import assert_close, oracle_layer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device():
    dev = CudaComputeDevice(0)
    yield dev
    dev.close()


def bf16(x):
    return synthetic.f32_to_bf16(np.asarray(x, dtype=np.float32))


def plan_of(device, **kw):
    fields = {"hidden": 256, "intermediate": 384, "experts": 8, "k": 2, "act_block": 32} | kw
    tokens = fields.pop("tokens", 64)
    return MoePlan(device, geometry_from_config(synthetic.MoeConfig("edges", **fields), tokens))


# one vector, a partial pass of the block, the longest row a block keeps, the first that it does not; the last count of
# short rows that goes to blocks and the first that goes to warps, the shortest row that always goes to blocks
@pytest.mark.parametrize("rows,hidden", [(3, 8), (2, 8200), (150, 1032), (2, 24544), (2, 24552), (2368, 72), (2369, 72),
                                         (2369, 2040), (2369, 2048)])
def test_rms_norm_rows(device, rows, hidden):
    rng = np.random.default_rng(hidden)
    x, w = bf16(rng.standard_normal((rows, hidden))), bf16(1.0 + 0.1 * rng.standard_normal(hidden))
    plan = plan_of(device)
    xb, wb, ob = device.resident_buffer_from(x), device.resident_buffer_from(w), device.create_resident_buffer(x.nbytes)
    plan.rms_norm(rows, hidden, xb, ob, wb, 1e-6, 0.0)
    np.testing.assert_array_equal(ob.read(np.uint16).reshape(x.shape), mo.rms_norm(x, w, 1e-6, 0.0))
    plan.destroy()


def test_dense_linears_of_one_shape_keep_their_own_tables(device):
    """Two matrices of one shape in turn, then one of them with new contents, then more matrices than are kept."""
    rng = np.random.default_rng(5)
    rows, cols, tokens = 128, 256, 9
    plan = plan_of(device)
    x = bf16(rng.standard_normal((tokens, cols)))
    xb, ob = device.resident_buffer_from(x), device.create_resident_buffer(tokens * rows * 2)
    mats = []
    for _ in range(67):
        w, s = rng.integers(0, 256, (rows, cols // 2), dtype=np.uint8), rng.integers(121, 128, (rows, cols // 32), dtype=np.uint8)
        mats.append([w, s, device.resident_buffer_from(w), device.resident_buffer_from(s)])

    def check(i):
        ob.fill(0)
        plan.dense_linear(tokens, xb, ob, mats[i][2], mats[i][3], rows, cols)
        assert_close(ob.read(np.uint16).reshape(tokens, rows), mo.dense_linear_mxfp4(x, mats[i][0], mats[i][1], 32, tier=1))

    for i in (0, 1, 0, 1):
        check(i)
    mats[1][1] = rng.integers(121, 128, (rows, cols // 32), dtype=np.uint8)
    mats[1][3].write_bytes(mats[1][1])
    for i in (1, 0, *range(2, 67), 0, 1, 66):
        check(i)
    assert plan.status() == 0
    plan.destroy()


# routes on either side of the one-block schedule's single pass (1024) and of its limit (1280), whole and ragged blocks of 256 routes, both scale
# blocks, a K tail (352 = 2.75 x 128), an expert that is not resident
@pytest.mark.parametrize("name,shape,tokens,absent", [
    ("gpt-oss-20b", (256, 384, 16), 256, None), ("gpt-oss-20b", (352, 160, 33), 257, 5), ("gpt-oss-20b", (1056, 320, 16), 1100, 0),
    ("gpt-oss-20b", (256, 384, 16), 320, 3), ("gpt-oss-20b", (352, 160, 33), 321, 5), ("deepseek-v3", (256, 256, 24), 143, 24),
    ("deepseek-v3", (512, 256, 24), 113, None), ("deepseek-v3", (384, 640, 24), 114, 24), ("deepseek-v3", (1024, 256, 256), 512, 7)])
def test_layer_call_equals_its_nodes(device, name, shape, tokens, absent):
    """The layer call schedules, quantises and fuses in its own way; the node operators are the plain one."""
    cfg = synthetic.small_variant(synthetic.CONFIGS[name], *shape)
    case = synthetic.make_case(cfg, tokens, seed=3)
    plan = MoePlan.for_config(device, cfg, tokens)
    bank = ExpertBank.upload(device, case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)
    if absent is not None:
        for slots, params in ((bank.gate_up_slots, 4), (bank.down_slots, 2)):
            words = slots.read(np.uint32).copy()
            words[absent * params:(absent + 1) * params] = 0xffffffff
            slots.write_bytes(words)
    hidden, rw = device.resident_buffer_from(case.hidden), device.resident_buffer_from(case.router_w)
    rb = device.resident_buffer_from(case.router_bias) if case.router_bias is not None else None
    sb = device.resident_buffer_from(case.select_bias) if case.select_bias is not None else None
    K, H = cfg.total_k, cfg.hidden
    make = device.create_resident_buffer
    out, want, routes = make(tokens * H * 2), make(tokens * H * 2), make(tokens * K * 4)
    plan.layer(tokens, bank, hidden, out, router_weights=rw, router_bias=rb, bias=sb, routes_out=routes)
    missed = plan.status()
    frames, outputs, gate, down = make(tokens * plan.frame_words * 4), make(tokens * K * H * 2), make(28), make(28)
    frames.fill(0)
    outputs.fill(0)
    control = np.array([tokens, 0, 0, 0, 0, 0, 0], dtype=np.uint32)
    gate.write_bytes(control)
    down.write_bytes(control)
    plan.moe_route_compact(tokens, routes, frames, gate, bank.gate_up_slots)
    plan.independent_sparse_moe_gate_up(tokens, hidden, routes, frames, bank.gate_up_addresses, bank.gate_up_slots, gate)
    plan.moe_route_count(tokens, routes, down, bank.down_slots)
    plan.independent_sparse_moe_down(tokens, frames, routes, outputs, bank.down_addresses, bank.down_slots, down)
    plan.moe_reduce(tokens, outputs, want)
    np.testing.assert_array_equal(out.read(np.uint16), want.read(np.uint16))
    assert missed == plan.status() and (missed == 0) == (absent is None)
    plan.destroy()


# the 4 x 8 tiles with ragged tokens, an odd expert count and rows that end inside a step; the calls just below and above
# each limit of their rule (5, 8 and 9 blocks on each of 148 SMs); the tiled form with a row of less than one chunk and last chunks that end in their first or second half
@pytest.mark.parametrize("tokens,hidden,experts,bias", [(98, 288, 199, 1), (255, 1056, 74, 0), (94, 288, 192, 0), (257, 32, 17, 0),
                                                        (289, 288, 8, 1), (300, 352, 33, 0), (144, 96, 159, 1), (145, 96, 159, 0),
                                                        (145, 96, 255, 1), (149, 96, 255, 0), (164, 96, 255, 0), (165, 96, 255, 1)])
def test_router_projection_tiles(device, tokens, hidden, experts, bias):
    rng = np.random.default_rng(tokens + hidden)
    plan = plan_of(device, tokens=tokens, hidden=hidden, experts=experts)
    x, w = bf16(rng.standard_normal((tokens, hidden))), bf16(0.1 * rng.standard_normal((experts, hidden)))
    b = bf16(rng.standard_normal(experts)) if bias else None
    out = device.create_resident_buffer(tokens * ((experts + 1) // 2) * 4)
    plan.linear(tokens, device.resident_buffer_from(x), out, device.resident_buffer_from(w),
                device.resident_buffer_from(b) if bias else None)
    np.testing.assert_array_equal(out.read(np.uint32).reshape(tokens, -1), mo.linear_bf16(x, w, b))
    plan.destroy()


# the tiled form beyond its ring of four chunks of 512 columns: rows of whole chunks, rows that end in each quarter of one and
# inside a step, ragged token and output tiles; subnormal inputs count in full
@pytest.mark.parametrize("tokens,hidden,experts", [(257, 2560, 16), (261, 2592, 18), (257, 2880, 32), (290, 4992, 5), (257, 2432, 17)])
def test_router_projection_long_rows(device, tokens, hidden, experts):
    rng = np.random.default_rng(tokens + hidden)
    plan = plan_of(device, tokens=tokens, hidden=hidden, experts=experts)
    x, w = bf16(rng.standard_normal((tokens, hidden))), bf16(0.1 * rng.standard_normal((experts, hidden)))
    x[:, ::7], w[0] = x[:, ::7] & 0x807F, w[0] & 0x807F
    out = device.create_resident_buffer(tokens * ((experts + 1) // 2) * 4)
    plan.linear(tokens, device.resident_buffer_from(x), out, device.resident_buffer_from(w), None)
    np.testing.assert_array_equal(out.read(np.uint32).reshape(tokens, -1), mo.linear_bf16(x, w, None))
    plan.destroy()


# groups of one expert, of two (less than a warp of experts), of 16 and of 32, one beyond the lanes (the shared-memory
# form), every group kept; logits with ties, infinities and NaN
@pytest.mark.parametrize("experts,n_group,topk_group,k", [(24, 24, 5, 4), (16, 8, 3, 4), (128, 8, 4, 6), (256, 8, 4, 8), (256, 8, 8, 8),
                                                          (64, 1, 1, 3), (256, 4, 2, 8)])
@pytest.mark.parametrize("activation", [synthetic.ACT_SIGMOID, synthetic.ACT_SOFTMAX])
def test_group_limited_routing(device, experts, n_group, topk_group, k, activation):
    cfg = synthetic.MoeConfig("groups", 256, 256, experts, k, activation=activation, n_group=n_group, topk_group=topk_group,
                              always_count=1, bias_dtype=synthetic.BIAS_F32, act_block=32)
    rng = np.random.default_rng(experts + n_group)
    tokens = 61
    logits = np.round(2.0 * rng.standard_normal((tokens, experts))).astype(np.float32)
    if activation == synthetic.ACT_SIGMOID:
        logits[3, ::3], logits[4, 1::5], logits[5, :2] = np.inf, -np.inf, np.nan
    bias = np.round(2.0 * rng.standard_normal(experts)).astype(np.float32) / 8
    bias[:2] = 0.0
    words = bf16(logits).view(np.uint32)
    plan = MoePlan.for_config(device, cfg, tokens)
    routes = device.create_resident_buffer(tokens * cfg.total_k * 4)
    plan.moe_route(tokens, device.resident_buffer_from(words), routes, device.resident_buffer_from(bias), None)
    want, _ = mo.route(mo.router_params_from(cfg), words, bias)
    np.testing.assert_array_equal(routes.read(np.uint32).reshape(want.shape), want)
    plan.destroy()


# the last batch that is routed and scheduled in one launch and the first that is not; fewer warps of routes than of
# tokens and the other way round; one and four experts a lane; an expert count beyond it
@pytest.mark.parametrize("name,experts,tokens", [("gpt-oss-20b", 32, 1), ("gpt-oss-20b", 33, 9), ("gpt-oss-20b", 128, 17),
                                                 ("gpt-oss-20b", 128, 16), ("gpt-oss-20b", 33, 16), ("gpt-oss-20b", 33, 17),
                                                 ("gpt-oss-20b", 16, 32), ("gpt-oss-20b", 16, 33), ("tiny", 8, 32),
                                                 ("gpt-oss-20b", 129, 8)])
def test_layer_routes_equal_the_router_node(device, name, experts, tokens):
    cfg = synthetic.small_variant(synthetic.CONFIGS[name], 256, 256, experts)
    case = synthetic.make_case(cfg, tokens, seed=7)
    plan = MoePlan.for_config(device, cfg, tokens)
    bank = ExpertBank.upload(device, case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)
    hidden, rw = device.resident_buffer_from(case.hidden), device.resident_buffer_from(case.router_w)
    rb = device.resident_buffer_from(case.router_bias) if case.router_bias is not None else None
    make = device.create_resident_buffer
    out, routes, want = make(tokens * cfg.hidden * 2), make(tokens * cfg.total_k * 4), make(tokens * cfg.total_k * 4)
    logits, counts, want_counts = make(tokens * ((experts + 1) // 2) * 4), make(plan.telemetry_words() * 4), make(plan.telemetry_words() * 4)
    counts.fill(0)
    want_counts.fill(0)
    plan.layer(tokens, bank, hidden, out, router_weights=rw, router_bias=rb, routes_out=routes, telemetry=counts)
    plan.linear(tokens, hidden, logits, rw, rb)
    plan.moe_route(tokens, logits, want, None, want_counts)
    np.testing.assert_array_equal(routes.read(np.uint32), want.read(np.uint32))
    np.testing.assert_array_equal(counts.read(np.uint32), want_counts.read(np.uint32))
    assert_close(out.read(np.uint16).reshape(tokens, -1), oracle_layer(case)["output"])
    assert plan.status() == 0
    plan.destroy()


def test_layer_of_rows_off_the_16_byte_grid(device):
    """Hidden rows that the token-wise quantisation cannot read take the general one: the same result."""
    cfg = synthetic.small_variant(synthetic.CONFIGS["gpt-oss-20b"], 256, 320, 16)
    tokens = 40
    case = synthetic.make_case(cfg, tokens, seed=11)
    plan = MoePlan.for_config(device, cfg, tokens)
    bank = ExpertBank.upload(device, case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)
    rw, rb = device.resident_buffer_from(case.router_w), device.resident_buffer_from(case.router_bias)
    room = device.create_resident_buffer(case.hidden.nbytes + 16)
    results = []
    for shift in (0, 8):
        room.write_bytes(case.hidden, shift)
        hidden = ResidentBuffer.wrap(device, room.device_address() + shift, case.hidden.nbytes)
        out = device.create_resident_buffer(tokens * cfg.hidden * 2)
        plan.layer(tokens, bank, hidden, out, router_weights=rw, router_bias=rb)
        results.append(out.read(np.uint16))
        hidden.destroy()
    np.testing.assert_array_equal(results[0], results[1])
    assert plan.status() == 0
    plan.destroy()


@pytest.mark.parametrize("path", [1, 2])
def test_dense_linear_refuses_matrices_off_the_32_byte_grid(device, path):
    rows, cols, tokens = 128, 256, 5
    rng = np.random.default_rng(3)
    plan = plan_of(device)
    plan.set_expert_path(path)
    x = bf16(rng.standard_normal((tokens, cols)))
    w, s = rng.integers(0, 256, (rows, cols // 2), dtype=np.uint8), rng.integers(121, 128, (rows, cols // 32), dtype=np.uint8)
    xb, ob = device.resident_buffer_from(x), device.create_resident_buffer(tokens * rows * 2)
    wroom, sroom = device.create_resident_buffer(w.nbytes + 32), device.create_resident_buffer(s.nbytes + 32)
    wroom.write_bytes(w), sroom.write_bytes(s)

    def at(room, shift, array):
        return ResidentBuffer.wrap(device, room.device_address() + shift, array.nbytes)

    for weights, scales in ((at(wroom, 16, w), at(sroom, 0, s)), (at(wroom, 0, w), at(sroom, 4, s))):
        with pytest.raises(CudaError):
            plan.dense_linear(tokens, xb, ob, weights, scales, rows, cols)
    plan.dense_linear(tokens, xb, ob, at(wroom, 0, w), at(sroom, 0, s), rows, cols)
    assert_close(ob.read(np.uint16).reshape(tokens, rows), mo.dense_linear_mxfp4(x, w, s, 32, tier=1))
    plan.destroy()


# rows of scale bytes of an odd count (352 / 32), an even one (320 / 32) and whole words (1152 / 32), K blocks in one, one and
# three groups of four
@pytest.mark.parametrize("path,cols", [(1, 352), (2, 352), (2, 320), (2, 1152)])
@pytest.mark.parametrize("handles", ["kept", "fresh"])
def test_dense_scales_rewritten_behind_wrapped_handles(device, path, cols, handles):
    """Two matrices of one shape in turn, their memory the caller's own: codes and scales are refilled in place, without
    a word to the library, through the handles that were used before or through new ones. Every call reads what is there."""
    rows, tokens = 160, 9
    rng = np.random.default_rng(17)
    plan = plan_of(device)
    plan.set_expert_path(path)
    x = bf16(rng.standard_normal((tokens, cols)))
    xb, ob = device.resident_buffer_from(x), device.create_resident_buffer(tokens * rows * 2)
    rooms = [[device.create_resident_buffer(rows * cols // 2), device.create_resident_buffer(rows * cols // 32)] for _ in range(2)]

    def wrapped(i):
        return [ResidentBuffer.wrap(device, room.device_address(), room.byte_capacity) for room in rooms[i]]

    kept = [wrapped(0), wrapped(1)]
    for which in (0, 1, 0, 1, 1, 0, 0):
        w, s = rng.integers(0, 256, (rows, cols // 2), dtype=np.uint8), rng.integers(118, 128, (rows, cols // 32), dtype=np.uint8)
        rooms[which][0].write_bytes(w), rooms[which][1].write_bytes(s)
        plan.dense_linear(tokens, xb, ob, *(kept[which] if handles == "kept" else wrapped(which)), rows, cols)
        assert_close(ob.read(np.uint16).reshape(tokens, rows), mo.dense_linear_mxfp4(x, w, s, 32, tier=1))
    assert plan.status() == 0
    plan.destroy()


# the gate/up epilogue makes the down operands (scale blocks of 32 and 128 rows), or a pass over the frames does (blocks of
# 64, hidden rows off the 16-byte grid, the CUDA-core path)
@pytest.mark.parametrize("path,block,shift", [(2, 32, 0), (2, 32, 8), (2, 64, 0), (2, 128, 0), (2, 128, 8), (1, 32, 0)])
@pytest.mark.parametrize("tokens", [37, 900])  # one-block and three-launch schedule
def test_routes_without_gate_up_count_as_zeros(device, path, block, shift, tokens):
    """An expert absent from the gate/up tables alone, after a call that had every expert: its routes give what they give
    when it is absent from both tables, rows of zeros, and not what the earlier call left in the plan's frames."""
    cfg = synthetic.MoeConfig("zeros", hidden=256, intermediate=384, experts=8, k=2, act_block=block)
    case = synthetic.make_case(cfg, tokens, seed=23)
    plan = MoePlan.for_config(device, cfg, tokens)
    plan.set_expert_path(path)
    bank = ExpertBank.upload(device, case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)
    room, rw = device.create_resident_buffer(case.hidden.nbytes + 16), device.resident_buffer_from(case.router_w)
    room.write_bytes(case.hidden, shift)
    hidden = ResidentBuffer.wrap(device, room.device_address() + shift, case.hidden.nbytes)
    out = device.create_resident_buffer(tokens * cfg.hidden * 2)

    def call():
        plan.layer(tokens, bank, hidden, out, router_weights=rw)
        return out.read(np.uint16)

    def drop(slots, params):
        words = slots.read(np.uint32).copy()
        words[3 * params:4 * params] = 0xffffffff
        slots.write_bytes(words)

    whole = call()
    drop(bank.gate_up_slots, 4)
    got = call()
    drop(bank.down_slots, 2)
    want = call()
    assert not np.array_equal(whole, want)
    np.testing.assert_array_equal(got, want)
    plan.destroy()


# one step of four, a whole second one, the nine that are taken at once and the counts beside it, remainders beyond
@pytest.mark.parametrize("k", [3, 8, 9, 10, 13, 18])
@pytest.mark.parametrize("scale", [1.0, 2.5])
def test_combine_of_any_route_count(device, k, scale):
    tokens = 37
    cfg = synthetic.MoeConfig("combine", hidden=288, intermediate=256, experts=32, k=k, act_block=32)
    geometry = geometry_from_config(cfg, tokens)
    geometry.reduce_scale = scale
    plan = MoePlan(device, geometry)
    rows = bf16(np.random.default_rng(k).standard_normal((tokens, k, cfg.hidden)))
    out = device.create_resident_buffer(tokens * cfg.hidden * 2)
    plan.moe_reduce(tokens, device.resident_buffer_from(rows), out)
    np.testing.assert_array_equal(out.read(np.uint16).reshape(tokens, cfg.hidden), mo.reduce(rows, tokens, k, cfg.hidden, scale))
    plan.destroy()


# 16- and 32-token tiles in row pairs: enough experts for six rounds of the SMs (min(routes, experts) x 8 row pairs >= 888),
# a last pair that is a lone 128-row half (1920 = 7.5 x 256), a K tail (352 = 2.75 x 128), a native FP8 resource
@pytest.mark.parametrize("name,shape,tokens,native", [("gpt-oss-20b", (1920, 352, 128), 250, 0), ("gpt-oss-20b", (1920, 352, 128), 620, 0),
                                                      ("deepseek-v3", (1920, 384, 128), 100, 1), ("deepseek-v3", (1920, 384, 128), 300, 1)])
def test_narrow_row_pairs_match_the_checker(device, name, shape, tokens, native):
    cfg = synthetic.replace(synthetic.small_variant(synthetic.CONFIGS[name], *shape), native_fp8_resources=native)
    assert min(tokens * cfg.total_k, cfg.total_experts) * -(-cfg.hidden // 256) >= 6 * 148
    case = synthetic.make_case(cfg, tokens, seed=13)
    tensors = [list(t) for t in (case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)]
    for e in range(cfg.total_experts - native, cfg.total_experts):
        for i, t in enumerate(synthetic.native_fp8_tensors(cfg, 13, e)):
            tensors[i][e] = t
    plan = MoePlan.for_config(device, cfg, tokens)
    plan.set_expert_path(2)
    bank = ExpertBank.upload(device, *tensors)
    out = device.create_resident_buffer(tokens * cfg.hidden * 2)
    plan.layer(tokens, bank, device.resident_buffer_from(case.hidden), out, router_weights=device.resident_buffer_from(case.router_w),
               router_bias=device.resident_buffer_from(case.router_bias) if case.router_bias is not None else None,
               bias=device.resident_buffer_from(case.select_bias) if case.select_bias is not None else None)
    logits = mo.linear_bf16(case.hidden, case.router_w, case.router_bias)
    sample = sampled.sample_tokens(tokens, 96, seed=tokens)
    want = sampled.layer_on_sample(cfg, case.hidden, logits, case.select_bias, sample, lambda e: [t[e] for t in tensors])
    assert_close(out.read(np.uint16).reshape(tokens, cfg.hidden)[sample], want["output"], f"{name} narrow row pairs T{tokens}")
    assert plan.status() == 0
    plan.destroy()
    bank.destroy()


# one CTA's tiles with tensor maps, by width (16, 32, 64, 96 tokens): K of whole pairs of blocks, of a lone block after them, of
# a trailing half block after either, of a single block; rows that end inside a tile; a native FP8 resource; and 16- and
# 32-token tiles in row pairs (tall boxes) with a last pair that is a lone half
@pytest.mark.parametrize("name,shape,tokens,native", [
    ("gpt-oss-20b", (576, 320, 16), 9, 0), ("gpt-oss-20b", (704, 448, 16), 60, 0), ("gpt-oss-20b", (384, 128, 16), 150, 0),
    ("gpt-oss-20b", (128, 192, 16), 340, 0), ("gpt-oss-20b", (448, 576, 16), 48, 0), ("deepseek-v3", (512, 384, 16), 5, 0),
    ("deepseek-v3", (384, 640, 16), 33, 1), ("deepseek-v3", (640, 256, 16), 150, 1), ("gpt-oss-20b", (1920, 448, 128), 250, 0),
    ("deepseek-v3", (1920, 384, 128), 300, 1)])
def test_tiles_by_tensor_map_match_the_checker(device, name, shape, tokens, native):
    cfg = synthetic.replace(synthetic.small_variant(synthetic.CONFIGS[name], *shape), native_fp8_resources=native)
    assert tokens * cfg.total_k <= 96 * cfg.total_experts
    case = synthetic.make_case(cfg, tokens, seed=19)
    tensors = [list(t) for t in (case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)]
    for e in range(cfg.total_experts - native, cfg.total_experts):
        for i, t in enumerate(synthetic.native_fp8_tensors(cfg, 19, e)):
            tensors[i][e] = t
    plan = MoePlan.for_config(device, cfg, tokens)
    plan.set_expert_path(2)
    bank = ExpertBank.upload(device, *tensors)
    out = device.create_resident_buffer(tokens * cfg.hidden * 2)
    plan.layer(tokens, bank, device.resident_buffer_from(case.hidden), out, router_weights=device.resident_buffer_from(case.router_w),
               router_bias=device.resident_buffer_from(case.router_bias) if case.router_bias is not None else None,
               bias=device.resident_buffer_from(case.select_bias) if case.select_bias is not None else None)
    logits = mo.linear_bf16(case.hidden, case.router_w, case.router_bias)
    sample = sampled.sample_tokens(tokens, 64, seed=tokens)
    want = sampled.layer_on_sample(cfg, case.hidden, logits, case.select_bias, sample, lambda e: [t[e] for t in tensors])
    assert_close(out.read(np.uint16).reshape(tokens, cfg.hidden)[sample], want["output"], f"{name} {shape} one CTA T{tokens}")
    assert plan.status() == 0
    plan.destroy()
    bank.destroy()


# the input quantised beside the matrix (scale blocks of 32 and 128, a ragged last 512 columns) and in a launch of its own
# (blocks of 64, rows off the 16-byte grid); several row tiles with a ragged last one, a row beyond one token tile
@pytest.mark.parametrize("block,shift,rows,cols,tokens", [(32, 0, 288, 544, 5), (32, 0, 160, 1056, 131), (128, 0, 384, 640, 33),
                                                         (64, 0, 320, 576, 17), (32, 8, 288, 544, 17), (128, 8, 256, 640, 200)])
def test_dense_linear_operands(device, block, shift, rows, cols, tokens):
    rng = np.random.default_rng(rows + cols)
    plan = plan_of(device, act_block=block, tokens=256)
    plan.set_expert_path(2)
    x = bf16(rng.standard_normal((tokens, cols)))
    w, s = rng.integers(0, 256, (rows, cols // 2), dtype=np.uint8), rng.integers(118, 128, (rows, cols // 32), dtype=np.uint8)
    room, ob = device.create_resident_buffer(x.nbytes + 16), device.create_resident_buffer(tokens * rows * 2)
    room.write_bytes(x, shift)
    xb = ResidentBuffer.wrap(device, room.device_address() + shift, x.nbytes)
    plan.dense_linear(tokens, xb, ob, device.resident_buffer_from(w), device.resident_buffer_from(s), rows, cols)
    assert_close(ob.read(np.uint16).reshape(tokens, rows), mo.dense_linear_mxfp4(x, w, s, block, tier=1))
    assert plan.status() == 0
    plan.destroy()


# matrices of so many rows that their 16-token tiles take two row tiles at a time: the last that do not (73 pairs of 128 rows), the first, with
# a lone last half, and whole pairs; a K tail
@pytest.mark.parametrize("rows,cols,tokens", [(18688, 352, 12), (18720, 352, 12), (18944, 256, 3), (18944, 128, 1)])
def test_dense_linear_of_many_rows(device, rows, cols, tokens):
    rng = np.random.default_rng(rows + cols)
    plan = plan_of(device, act_block=32, tokens=16)
    x = bf16(rng.standard_normal((tokens, cols)))
    w, s = rng.integers(0, 256, (rows, cols // 2), dtype=np.uint8), rng.integers(118, 128, (rows, cols // 32), dtype=np.uint8)
    ob = device.create_resident_buffer(tokens * rows * 2)
    plan.dense_linear(tokens, device.resident_buffer_from(x), ob, device.resident_buffer_from(w), device.resident_buffer_from(s), rows, cols)
    assert_close(ob.read(np.uint16).reshape(tokens, rows), mo.dense_linear_mxfp4(x, w, s, 32, tier=1))
    assert plan.status() == 0
    plan.destroy()


# every token tile from one plan: a call has the tensor maps of its tile whatever the plan's largest call is (boxes of one K
# block and of two, whole pairs of blocks and a trailing half; one-byte weights)
@pytest.mark.parametrize("name,shape,native", [("gpt-oss-20b", (576, 512, 8), 0), ("deepseek-v3", (512, 384, 16), 1)])
def test_calls_of_every_tile_from_one_plan(device, name, shape, native):
    cfg = synthetic.replace(synthetic.small_variant(synthetic.CONFIGS[name], *shape), native_fp8_resources=native)
    case = synthetic.make_case(cfg, 500, seed=23)
    tensors = [list(t) for t in (case.w1, case.s1, case.w3, case.s3, case.w2, case.s2)]
    for e in range(cfg.total_experts - native, cfg.total_experts):
        for i, t in enumerate(synthetic.native_fp8_tensors(cfg, 23, e)):
            tensors[i][e] = t
    bank = ExpertBank.upload(device, *tensors)
    hidden, rw = device.resident_buffer_from(case.hidden), device.resident_buffer_from(case.router_w)
    args = {"router_weights": rw, "router_bias": device.resident_buffer_from(case.router_bias) if case.router_bias is not None else None,
            "bias": device.resident_buffer_from(case.select_bias) if case.select_bias is not None else None}
    out = device.create_resident_buffer(500 * cfg.hidden * 2)
    large = MoePlan.for_config(device, cfg, 500)
    for tokens in (1, 9, 10, 20, 40, 80, 96, 200, 500):
        own = MoePlan.for_config(device, cfg, tokens)
        got = []
        for plan in (large, own):
            plan.set_expert_path(2)
            out.fill(0)
            plan.layer(tokens, bank, hidden, out, **args)
            assert plan.status() == 0
            got.append(out.read(np.uint16))
        np.testing.assert_array_equal(got[0], got[1], err_msg=f"{tokens} tokens")
        own.destroy()
    large.destroy()
    bank.destroy()


# few blocks of long rows, whose loads run 24 steps of 128 columns ahead: either side of the lines of the rule (148 and 592 blocks of 2 tokens x
# 4 outputs, 1024 and 2048 columns), rows that end inside a step, with and beyond the first 24
@pytest.mark.parametrize("tokens,hidden,experts", [(73, 1056, 16), (75, 1056, 16), (1, 1024, 30), (75, 2048, 16), (75, 2080, 16), (255, 3072, 16),
                                                   (255, 3104, 15), (2, 6176, 5), (236, 2080, 19), (238, 2080, 19)])
def test_router_projection_of_few_blocks(device, tokens, hidden, experts):
    rng = np.random.default_rng(tokens + hidden)
    plan = plan_of(device, tokens=tokens, hidden=hidden, experts=experts)
    x, w = bf16(rng.standard_normal((tokens, hidden))), bf16(0.1 * rng.standard_normal((experts, hidden)))
    x[0] = 0x8000  # (sums of minus zero, which a step past the end would turn into zero)
    w[1] &= 0x7FFF
    out = device.create_resident_buffer(tokens * ((experts + 1) // 2) * 4)
    plan.linear(tokens, device.resident_buffer_from(x), out, device.resident_buffer_from(w), None)
    np.testing.assert_array_equal(out.read(np.uint32).reshape(tokens, -1), mo.linear_bf16(x, w, None))
    plan.destroy()
