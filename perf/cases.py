"""The work a runtime has this library do, as measured cases.

A model server holds one device, mounts every MoE layer as a plan plus resident expert weights, and then calls
the layer once per layer and step: on a handful of tokens while decoding, on hundreds when requests share a step,
on thousands while it reads prompts. Four kinds of call cover that:

  layer   one `MoePlan.layer` call on buffers that are resident on the GPU
  host    one `MoePlan.layer_host` call: tokens from page-locked host memory, the result back in it
  nodes   the same layer walked one operator at a time, as a runtime does that steps through a node list
  ffn     the dense feed-forward block beside the experts: norm, gate and up, SiLU, down, residual add

Shapes are those of `nerve_b200.synthetic.CONFIGS` and generic ones; weights and activations are drawn on the GPU
with the distributions of that module. A state owns its own weights, so successive passes over different states read
different bytes, as the successive layers of a model do.
"""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import torch

from nerve_b200 import synthetic
from nerve_b200.backend import CudaComputeDevice, ExpertBank, MoePlan, ResidentBuffer, geometry_from_config

_DEVICE = None


def _device() -> CudaComputeDevice:
    """The one device object of the process."""
    global _DEVICE
    if _DEVICE is None:
        torch.cuda.init()
        _DEVICE = CudaComputeDevice(0)
    return _DEVICE


# ---- the cases ---------------------------------------------------------------------------------------------

def listed() -> list[dict]:
    return [
        # the smallest layer there is: nothing but launches and latency
        {"name": "tiny_64", "kind": "layer", "config": "tiny", "tokens": 64},
        # one user decoding: four experts of 32, one token
        {"name": "decode_1", "kind": "layer", "config": "gpt-oss-20b", "tokens": 1},
        # a few users decoding: about two thirds of the experts, one token each
        {"name": "decode_7", "kind": "layer", "config": "gpt-oss-20b", "tokens": 7},
        # a full decode batch: every expert's weights cross memory once
        {"name": "decode_64", "kind": "layer", "config": "gpt-oss-20b", "tokens": 64},
        # a decode step whose activations live on the host
        {"name": "host_32", "kind": "host", "config": "gpt-oss-20b", "tokens": 32},
        # a decode step of a runtime that walks the node list
        {"name": "nodes_45", "kind": "nodes", "config": "gpt-oss-20b", "tokens": 45},
        # decode requests and a prompt chunk in one step
        {"name": "mixed_501", "kind": "layer", "config": "gpt-oss-120b", "tokens": 501},
        # reading prompts, with the skewed expert load that real routers show
        {"name": "prefill_4096", "kind": "layer", "config": "gpt-oss-20b-prefill", "tokens": 4096},
        # reading prompts through a layer of many experts
        {"name": "prefill_8192", "kind": "layer", "config": "gpt-oss-120b", "tokens": 8192},
        # decoding through a wide layer: grouped routing, a shared expert kept in native FP8
        {"name": "wide_decode_96", "kind": "layer", "config": "deepseek-v3", "tokens": 96, "native": 1},
        # reading prompts through the wide layer: the largest call
        {"name": "wide_prefill_16384", "kind": "layer", "config": "deepseek-v3", "tokens": 16384},
        # a dense feed-forward block over a prompt chunk
        {"name": "ffn_777", "kind": "ffn", "config": "deepseek-v3", "tokens": 777},
    ]


_MAX_TOKENS = {"tiny": 4096, "gpt-oss-20b": 8192, "gpt-oss-20b-prefill": 8192, "gpt-oss-120b": 8192, "deepseek-v3": 16384}


def _log_uniform(rng, low: int, high: int) -> int:
    return max(low, min(high, round(low * (high / low) ** rng.random())))


def draw(rng) -> dict:
    kind = rng.choices(("layer", "host", "nodes", "ffn"), (60, 12, 14, 14))[0]
    case = {"kind": kind}
    if rng.random() < 0.7:
        case["config"] = rng.choice(sorted(_MAX_TOKENS))
    else:
        # a layer of another model: any multiple of 64, the routing rules of one of the two router families
        case["config"] = rng.choice(("gpt-oss-20b", "deepseek-v3"))
        case["hidden"] = 64 * _log_uniform(rng, 6, 64)
        case["intermediate"] = 64 * _log_uniform(rng, 4, 48)
        case["experts"] = rng.choice((16, 24, 32, 64, 96, 128))
    # (the activation block of the wide layer is 128 columns: one-byte weights need whole blocks too)
    if kind != "ffn" and case["config"] == "deepseek-v3" and rng.random() < 0.3 and all(
            case.get(k, 128) % 128 == 0 for k in ("hidden", "intermediate")):
        case["native"] = 1
    most = _MAX_TOKENS[case["config"]]
    case["tokens"] = _log_uniform(rng, 1, {"layer": most, "host": min(most, 1024), "nodes": min(most, 2048),
                                           "ffn": min(most, 8192)}[kind])
    return case


def _config(case: dict) -> synthetic.MoeConfig:
    cfg = synthetic.CONFIGS[case["config"]]
    if "hidden" in case:
        cfg = synthetic.small_variant(cfg, case["hidden"], case["intermediate"], case["experts"])
        whole = cfg.hidden % 128 == 0 and cfg.intermediate % 128 == 0
        cfg = replace(cfg, act_block=cfg.act_block if whole else 32, zipf_s=0.0)
    return replace(cfg, native_fp8_resources=case.get("native", 0))


# ---- inputs ------------------------------------------------------------------------------------------------

class State:
    """Inputs, weights, plan and output buffers of one case; everything is given back with the object."""

    def __init__(self, case: dict, seed: int):
        self.case, self.cfg, self.device = case, _config(case), _device()
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.handles, self.bank = [], None
        self.plan = MoePlan(self.device, geometry_from_config(self.cfg, case["tokens"]))

    def __del__(self):
        if getattr(self, "plan", None) is None:
            return
        self.device.synchronize()
        self.plan.destroy()
        self.plan = None
        if self.bank is not None:
            self.bank.destroy()
        for handle in self.handles:
            handle.destroy()

    def wrap(self, tensor: torch.Tensor) -> ResidentBuffer:
        return ResidentBuffer.wrap(self.device, tensor.data_ptr(), tensor.numel() * tensor.element_size())

    def buffer(self, tensor: torch.Tensor) -> ResidentBuffer:
        handle = self.wrap(tensor)
        self.handles.append(handle)
        return handle

    def normal(self, *shape, scale=1.0, mean=0.0) -> torch.Tensor:
        return torch.randn(*shape, generator=self.gen, device="cuda").mul_(scale).add_(mean).to(torch.bfloat16)

    def codes(self, *shape) -> torch.Tensor:
        """Packed E2M1 pairs, uniform over the sixteen values."""
        count = int(np.prod(shape))
        words = torch.randint(-(1 << 63), (1 << 63) - 1, ((count + 7) // 8,), generator=self.gen, device="cuda")
        return words.view(torch.uint8)[:count].view(*shape)

    def scales(self, *shape, low=121, high=128) -> torch.Tensor:
        return torch.randint(low, high, shape, generator=self.gen, device="cuda", dtype=torch.uint8)

    def native_codes(self, rows: int, cols: int) -> torch.Tensor:
        """E4M3 bytes without the two NaN codes."""
        codes = self.codes(rows, cols)
        return torch.where((codes & 0x7F) == 0x7F, torch.full_like(codes, 0x38), codes)

    def experts(self) -> None:
        """The packaged tensors of every expert and the tables that name them."""
        cfg = self.cfg
        H, I, packed = cfg.hidden, cfg.intermediate, cfg.total_experts - cfg.native_fp8_resources
        shapes = ((I, H), (I, H), (H, I))  # w1, w3, w2
        self.weights = [(self.codes(packed, r, c // 2), self.scales(packed, r, c // 32)) for r, c in shapes]
        per_expert = [[self.wrap(t[e]) for pair in self.weights for t in pair] for e in range(packed)]
        for _ in range(cfg.native_fp8_resources):
            native = [(self.native_codes(r, c), self.scales(-(-r // 128), -(-c // 128), low=112, high=119)) for r, c in shapes]
            self.weights += native
            per_expert.append([self.wrap(t) for pair in native for t in pair])
        self.bank = ExpertBank.from_resident(self.device, per_expert)

    def router(self) -> dict:
        """The router's parameters, as `MoePlan.layer` names them."""
        cfg = self.cfg
        E = cfg.experts
        self.router_w = self.normal(E, cfg.hidden, scale=0.02)
        args = {"router_weights": self.buffer(self.router_w), "router_bias": None, "bias": None}
        if cfg.logit_bias:
            bias = 0.1 * torch.randn(E, generator=self.gen, device="cuda")
            if cfg.zipf_s > 0.0:
                rank = torch.argsort(torch.rand(E, generator=self.gen, device="cuda")).float() + 1.0
                share = rank ** -cfg.zipf_s
                bias = bias + torch.log(share / share.sum())
            self.router_bias = bias.to(torch.bfloat16)
            args["router_bias"] = self.buffer(self.router_bias)
        if cfg.bias_dtype == synthetic.BIAS_F32:
            self.select_bias = 0.05 * torch.randn(E, generator=self.gen, device="cuda")
            args["bias"] = self.buffer(self.select_bias)
        return args


def _empty(shape, dtype) -> torch.Tensor:
    return torch.zeros(shape, dtype=dtype, device="cuda")


def prepare(case: dict, seed: int) -> State:
    s = State(case, seed)
    cfg, T = s.cfg, case["tokens"]
    H, I, K = cfg.hidden, cfg.intermediate, cfg.total_k
    s.hidden = s.normal(T, H)
    s.output = _empty((T, H), torch.bfloat16)
    if case["kind"] == "ffn":
        s.norm_weight = s.normal(H, scale=0.05, mean=1.0)
        s.dense = [(s.codes(r, c // 2), s.scales(r, c // 32, high=126), r, c) for r, c in ((I, H), (I, H), (H, I))]
        s.normed, s.down = _empty((T, H), torch.bfloat16), _empty((T, H), torch.bfloat16)
        s.gate, s.up, s.act = (_empty((T, I), torch.bfloat16) for _ in range(3))
        s.b = {k: s.buffer(getattr(s, k)) for k in ("hidden", "output", "norm_weight", "normed", "down", "gate", "up", "act")}
        s.mats = [(s.buffer(w), s.buffer(sc), r, c) for w, sc, r, c in s.dense]
        torch.cuda.synchronize()
        return s
    s.experts()
    s.args = s.router()
    s.routes = _empty((T, K), torch.int32)
    s.telemetry = _empty((s.plan.telemetry_words(),), torch.int32)
    s.b = {k: s.buffer(getattr(s, k)) for k in ("hidden", "output", "routes", "telemetry")}
    s.args.update(routes_out=s.b["routes"], telemetry=s.b["telemetry"])
    if case["kind"] == "host":
        s.hidden_host = s.hidden.cpu().pin_memory()
        s.output_host = torch.zeros((T, H), dtype=torch.bfloat16).pin_memory()
        s.hidden_np = s.hidden_host.view(torch.int16).numpy().view(np.uint16)
        s.output_np = s.output_host.view(torch.int16).numpy().view(np.uint16)
    elif case["kind"] == "nodes":
        s.logits = _empty((T, (cfg.experts + 1) // 2), torch.int32)
        s.frames = _empty((T, s.plan.frame_words), torch.int32)
        s.expert_outputs = _empty((T, K, H), torch.bfloat16)
        s.gate_control, s.down_control = _empty((7,), torch.int32), _empty((7,), torch.int32)
        s.b.update({k: s.buffer(getattr(s, k)) for k in ("logits", "frames", "expert_outputs", "gate_control", "down_control")})
        s.control_words = np.array([T, 0, 0, 0, 0, 0, 0], dtype=np.uint32)
    torch.cuda.synchronize()
    return s


# ---- one pass ------------------------------------------------------------------------------------------------

def run(s: State) -> dict:
    return {"layer": _run_layer, "host": _run_host, "nodes": _run_nodes, "ffn": _run_ffn}[s.case["kind"]](s)


def _run_layer(s: State) -> dict:
    s.plan.layer(s.case["tokens"], s.bank, s.b["hidden"], s.b["output"], **s.args)
    return {"output": s.output, "routes": s.routes, "telemetry": s.telemetry}


def _run_host(s: State) -> dict:
    s.plan.layer_host(s.case["tokens"], s.bank, s.hidden_np, s.output_np, **s.args)
    return {"output": s.output_host, "routes": s.routes, "telemetry": s.telemetry}


def _run_nodes(s: State) -> dict:
    p, b, T, bank = s.plan, s.b, s.case["tokens"], s.bank
    p.linear(T, b["hidden"], b["logits"], s.args["router_weights"], s.args["router_bias"])
    p.moe_route(T, b["logits"], b["routes"], s.args["bias"], b["telemetry"])
    b["gate_control"].write_bytes(s.control_words)
    p.moe_route_compact(T, b["routes"], b["frames"], b["gate_control"], bank.gate_up_slots)
    p.independent_sparse_moe_gate_up(T, b["hidden"], b["routes"], b["frames"], bank.gate_up_addresses, bank.gate_up_slots,
                                     b["gate_control"])
    b["down_control"].write_bytes(s.control_words)
    p.moe_route_count(T, b["routes"], b["down_control"], bank.down_slots)
    p.independent_sparse_moe_down(T, b["frames"], b["routes"], b["expert_outputs"], bank.down_addresses, bank.down_slots,
                                  b["down_control"])
    p.moe_reduce(T, b["expert_outputs"], b["output"])
    return {"logits": s.logits, "routes": s.routes, "telemetry": s.telemetry, "gate_control": s.gate_control,
            "down_control": s.down_control, "schedule": s.frames[:, p.data_words:],
            "intermediates": s.frames.view(torch.bfloat16)[:, :2 * p.data_words], "expert_outputs": s.expert_outputs,
            "output": s.output}


def _run_ffn(s: State) -> dict:
    p, b, T, cfg = s.plan, s.b, s.case["tokens"], s.cfg
    p.rms_norm(T, cfg.hidden, b["hidden"], b["normed"], b["norm_weight"], 1e-6)
    p.dense_linear(T, b["normed"], b["gate"], *s.mats[0])
    p.dense_linear(T, b["normed"], b["up"], *s.mats[1])
    p.silu_multiply(T, cfg.intermediate, b["gate"], b["up"], b["act"], cfg.swiglu_limit)
    p.dense_linear(T, b["act"], b["down"], *s.mats[2])
    p.residual_add(T, cfg.hidden, b["hidden"], b["down"], b["output"])
    return {"normed": s.normed, "gate": s.gate, "up": s.up, "act": s.act, "down": s.down, "output": s.output}


# ---- what a pass cannot do without ---------------------------------------------------------------------------

def _experts_touched(cfg: synthetic.MoeConfig, tokens: int) -> int:
    """How many experts a batch of drawn tokens selects: the router's rule on logits of the drawn distribution. (A
    sigmoid router saturates on its best experts and its selection bias then decides, so it touches far fewer than
    uniform routing would.)"""
    rng = np.random.default_rng(cfg.experts)
    T, E = min(tokens, 2048), cfg.experts
    score = rng.standard_normal((T, E)) * (0.02 * cfg.hidden ** 0.5)
    if cfg.logit_bias:
        score += 0.1 * rng.standard_normal(E) - cfg.zipf_s * np.log(1.0 + rng.permutation(E))
    if cfg.activation == synthetic.ACT_SIGMOID:
        score = 1.0 / (1.0 + np.exp(-score))
    if cfg.bias_dtype != synthetic.BIAS_NONE:
        score += 0.05 * rng.standard_normal(E)
    if cfg.n_group:
        grouped = score.reshape(T, cfg.n_group, -1)
        best = np.sort(grouped, axis=2)[:, :, -2:].sum(axis=2)
        kept = np.argsort(np.argsort(-best, axis=1), axis=1) < cfg.topk_group
        score = np.where(kept[:, :, None], grouped, -np.inf).reshape(T, E)
    return len(np.unique(np.argpartition(-score, cfg.k - 1, axis=1)[:, :cfg.k])) + cfg.always_count


def work(case: dict) -> dict:
    cfg, T = _config(case), case["tokens"]
    H, I, E, K = cfg.hidden, cfg.intermediate, cfg.experts, cfg.total_k
    if case["kind"] == "ffn":
        rows = T * (4 * H + 3 * I) * 2  # hidden in; normed, down and output out; gate, up and act out
        return {"bytes": 3 * H * I * 17 // 32 + rows + 2 * H, "flops": 2.0 * T * 3 * H * I}
    weights = _experts_touched(cfg, T) * cfg.expert_weight_bytes + cfg.native_fp8_resources * 3 * H * I * 15 // 32
    data = 2 * T * H * 2 + E * H * 2 + T * K * 4
    if case["kind"] == "nodes":  # every node's output is the caller's
        data += T * E * 2 + T * K * (I + H) * 2 + T * K * 4
    return {"bytes": float(weights + data), "flops": 2.0 * T * K * 3 * H * I + 2.0 * T * E * H}


def tolerance(case: dict) -> dict:
    """Routing is exact in every word. Expert rows are bf16 sums of E4M3 x E2M1 products accumulated in f32 in no
    fixed order: the layer's own bound against its f64-accumulated form."""
    return {"rel": 5e-3, "max": 0.1, "differ": 0.0}
