"""The forward passes that users of this library run, as measurable cases.

A case is one call of ``MoELayer.forward_ptr`` (device pointers, caller's stream) or, with ``host``, of
``MoELayer.forward_host`` (page-locked host buffers, copies inside the call) on a layer whose weights lie on the
GPU.  The layers are the benchmark shapes of ``ffai_b200.synth``; ``tokens`` is the batch, ``max_tokens`` what the
handle was sized for (a server sizes one handle for its prefill chunk and decodes through it too).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from ffai_b200 import capi, synth
from ffai_b200.moe import MoELayer

PREFILL_CHUNK = 2048    # tokens a serving handle is sized for when its own batch is smaller


def _case(layer, tokens, bits=4, group_size=64, row_bias=0, skewed=False, residual=False, host=False, max_tokens=None):
    return {"layer": layer, "tokens": tokens, "max_tokens": max_tokens or max(tokens, PREFILL_CHUNK), "bits": bits,
            "group_size": group_size, "row_bias": row_bias, "skewed": skewed, "residual": residual, "host": host}


def listed():
    return [
        # one user's chat: a single token through the 32-expert layer of 2880 x 2880 projections, decode-only handle
        dict(_case("gptoss", 1, max_tokens=64), name="gptoss_decode_1"),
        # the same layer as its checkpoints arrive (MXFP4 transcoded: groups of 32, row biases), a handful of users
        dict(_case("gptoss", 8, group_size=32, row_bias=1), name="gptoss_g32_decode_8"),
        # a full decode batch: every expert is selected
        dict(_case("gptoss", 64), name="gptoss_decode_64"),
        # a prompt of odd length through that layer
        dict(_case("gptoss", 777, group_size=32, row_bias=1), name="gptoss_g32_prompt_777"),
        # the smallest real step: one token through many small experts, where launches and latency count
        dict(_case("qwen", 1), name="qwen_decode_1"),
        # a mixed batch between decode and prefill: six rows for each of 128 experts, block output added to its input
        dict(_case("qwen", 100, residual=True), name="qwen_mixed_100"),
        # 8-bit experts, the format chosen for quality, in a small decode batch
        dict(_case("qwen", 4, bits=8), name="qwen_8bit_decode_4"),
        # the prefill chunk of the 128-expert layer
        dict(_case("qwen", 2048), name="qwen_prefill_2048"),
        # 256 experts and a gated 8-bit shared expert: a small decode batch ...
        dict(_case("shared", 3), name="shared_decode_3"),
        # ... the long prefill with everything on the device ...
        dict(_case("shared", 8192, residual=True), name="shared_prefill_8192"),
        # ... and the same from and to host memory
        dict(_case("shared", 8192, host=True), name="shared_prefill_8192_host"),
        # the largest: a long batch whose routing is skewed (the first experts get most rows), 5-bit experts
        dict(_case("qwen", 16384, bits=5, skewed=True), name="qwen_5bit_skewed_16384"),
    ]


def draw(rng):
    """One more case: a listed layer, format and option, any batch size of its range."""
    kind = rng.choice(["gptoss", "gptoss_g32", "qwen", "qwen_bits", "shared", "shared"])
    most = {"gptoss": 4096, "gptoss_g32": 4096, "qwen": 8192, "qwen_bits": 16384, "shared": 8192}[kind]
    tokens = max(1, min(most, int(round(math.exp(rng.uniform(0.0, math.log(most)))))))
    if tokens > 64 and rng.random() < 0.7:
        tokens |= 1    # prompts have any length
    residual = rng.random() < 0.5
    host = tokens <= 8192 and rng.random() < 0.15
    # a handle for decode alone, or one that takes prefill chunks as well
    max_tokens = 64 if tokens <= 64 and kind != "qwen_bits" and rng.random() < 0.3 else None
    if kind == "gptoss_g32":
        return _case("gptoss", min(tokens, most), group_size=32, row_bias=1, residual=residual, host=host, max_tokens=max_tokens)
    if kind == "qwen_bits":
        return _case("qwen", min(tokens, most), bits=rng.choice([3, 5, 6, 8]), skewed=rng.random() < 0.5, residual=residual, host=host)
    return _case(kind, min(tokens, most), residual=residual, host=host, max_tokens=max_tokens)


def _spec(case) -> synth.LayerSpec:
    base = {"gptoss": synth.cfg2_gptoss, "qwen": synth.cfg3_qwen, "shared": synth.cfg4_shared}[case["layer"]]()
    spec = base.with_(expert_bits=case["bits"], expert_group_size=case["group_size"], expert_row_bias=case["row_bias"])
    return spec.with_(router_has_bias=1, zipf_s=1.1) if case["skewed"] else spec


class DeviceLayer:
    """Weights of one layer on the GPU, in the library's layout, with the value distributions of ``synth.make_layer``."""

    def __init__(self, spec: synth.LayerSpec, seed: int):
        self.spec = spec
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.t = {}
        H, I, E, s = spec.hidden, spec.intermediate, spec.n_experts, spec
        self._linear("gate", E, H, s.router_kind, s.router_group_size)
        if s.router_has_bias:
            bias = (torch.from_numpy(synth.zipf_router_bias(E, s.zipf_s, s.zipf_strength)).cuda() if s.zipf_s > 0
                    else 0.05 * self._normal(E))
            self.t["gate.bias"] = bias.to(torch.bfloat16)
        for name, n_out, n_in in (("gate_proj", I, H), ("up_proj", I, H), ("down_proj", H, I)):
            self._qproj("experts." + name, E, n_out, n_in, s.expert_bits, s.expert_group_size, s.expert_row_bias)
        if s.shared_intermediate:
            Is = s.shared_intermediate
            for name, n_out, n_in in (("gate_proj", Is, H), ("up_proj", Is, H), ("down_proj", H, Is)):
                self._qproj("shared_expert." + name, 1, n_out, n_in, s.shared_bits, s.shared_group_size, 0)
            self._linear("shared_expert_gate", 1, H, s.shared_gate_kind, s.shared_gate_group_size)

    def _normal(self, *shape):
        return torch.randn(*shape, device="cuda", generator=self.gen)

    def _uniform(self, *shape):
        return torch.rand(*shape, device="cuda", generator=self.gen)

    def _qproj(self, name, n, n_out, n_in, bits, group, row_bias):
        # uniform random words are uniform random codes at every bit width
        self.t[name + ".weight"] = torch.randint(-2**31, 2**31, (n, n_out, n_in * bits // 32), device="cuda",
                                                 dtype=torch.int32, generator=self.gen)
        g = n_in // group
        self.t[name + ".scales"] = ((0.005 + 0.015 * self._uniform(n, n_out, g)) * (15.0 / ((1 << bits) - 1))).to(torch.bfloat16)
        self.t[name + ".biases"] = (-0.1 + 0.2 * self._uniform(n, n_out, g)).to(torch.bfloat16)
        if row_bias:
            self.t[name + ".row_bias"] = (0.1 * self._normal(n, n_out)).to(torch.bfloat16)

    def _linear(self, name, n_out, n_in, kind, group):
        w = 0.02 * self._normal(n_out, n_in)
        if kind == capi.LINEAR_BF16:
            self.t[name + ".weight"] = w.to(torch.bfloat16)
            return
        # 8-bit affine, fitted to each group's range
        v = w.reshape(n_out, n_in // group, group)
        lo, hi = v.amin(-1), v.amax(-1)
        scale, bias = ((hi - lo) / 255.0).to(torch.bfloat16), lo.to(torch.bfloat16)
        q = ((v - bias.float()[..., None]) / scale.float()[..., None]).round().clamp(0, 255).to(torch.uint8)
        self.t[name + ".weight"] = q.reshape(n_out, n_in).view(torch.int32)
        self.t[name + ".scales"], self.t[name + ".biases"] = scale, bias

    def weights_struct(self, ep_rank: int = 0, ep_world: int = 1) -> capi.MoEWeights:
        def ptrs(name, last):
            return [self.t[name + k].data_ptr() if name + k in self.t else None for k in (".weight", ".scales", ".biases", last)]

        w = capi.MoEWeights()
        w.location = capi.MEM_DEVICE
        w.router = capi.Linear(*ptrs("gate", ".bias"))
        for proj in ("gate_proj", "up_proj", "down_proj"):
            setattr(w, proj, capi.QProj(*ptrs("experts." + proj, ".row_bias")))
            if self.spec.shared_intermediate:
                setattr(w, "shared_" + proj, capi.QProj(*ptrs("shared_expert." + proj, ".row_bias")))
        if self.spec.shared_intermediate:
            w.shared_gate = capi.Linear(*ptrs("shared_expert_gate", ".bias"))
        return w


def prepare(case, seed):
    spec = _spec(case)
    weights = DeviceLayer(spec, seed)
    layer = MoELayer(weights, case["max_tokens"])
    T, H = case["tokens"], spec.hidden
    x = weights._normal(T, H).to(torch.bfloat16)
    residual = weights._normal(T, H).to(torch.bfloat16) if case["residual"] else None
    state = {"case": case, "weights": weights, "layer": layer, "T": T}
    if case["host"]:
        pinned = [None if t is None else t.view(torch.int16).cpu().pin_memory() for t in (x, residual)]
        out = torch.zeros(T, H, dtype=torch.int16).pin_memory()
        state.update(x_pin=pinned[0], residual_pin=pinned[1], out_pin=out, out=out.view(torch.bfloat16),
                     x=pinned[0].numpy().view(np.uint16),
                     residual=None if residual is None else pinned[1].numpy().view(np.uint16),
                     out_np=out.numpy().view(np.uint16))
    else:
        state.update(x=x, residual=residual, out=torch.zeros(T, H, dtype=torch.bfloat16, device="cuda"))
    return state


def run(state):
    if state["case"]["host"]:
        state["layer"].forward_host(state["x"], residual=state["residual"], out=state["out_np"])
    else:
        residual = state["residual"]
        state["layer"].forward_ptr(state["x"].data_ptr(), state["T"], state["out"].data_ptr(),
                                   0 if residual is None else residual.data_ptr(), torch.cuda.current_stream().cuda_stream)
    return state["out"]


def work(case):
    spec, T = _spec(case), case["tokens"]
    # experts that some token selects: expert e is chosen by a token with probability k * share(e), at most 1
    share = np.full(spec.n_experts, 1.0 / spec.n_experts)
    if case["skewed"]:
        share = np.power(np.arange(1, spec.n_experts + 1, dtype=np.float64), -spec.zipf_s)
        share /= share.sum()
    distinct = float(np.sum(1.0 - (1.0 - np.minimum(1.0, spec.top_k * share)) ** T))
    rows = T * spec.hidden * 2.0 * (3 if case["residual"] else 2)
    shared = 0.0
    if spec.shared_intermediate:
        shared = 3.0 * spec.hidden * spec.shared_intermediate * spec.bytes_per_weight(spec.shared_bits, spec.shared_group_size)
    return {"bytes": distinct * spec.bytes_per_expert() + spec.router_bytes() + shared + rows,
            "flops": sum(spec.prefill_flops(T).values())}


def tolerance(case):
    # bf16 outputs; between two implementations the expert weights, the activation's result and the down product may
    # each be rounded to bf16 or kept in fp32, and each such rounding is 2**-9 (0.2 %) of its value.  max: twice the
    # 2e-2 that the repository's parity tests allow one implementation against the fp32 result.
    return {"rel": 5e-3, "max": 4e-2}
