"""Performance cases of the MatMulNBits library: what a program that serves a quantized model has it do.

A case is a dict of plain values. ``kind`` says which public entry point runs:

* ``node``     one MatMulNBits node on device tensors (``MatMulNBitsWeights.matmul_device``)
* ``layer``    the seven projections of a decoder layer (``tools.decoder_layer.DecoderLayerProjections``)
* ``operator`` the registered operator on host arrays, as an evaluator runs it (``MatMulNBitsSession``)

``m`` tokens, ``bits`` 4 or 8, ``block`` codes per scale, ``zp`` / ``bias`` optional operands, ``level`` the
operator's accuracy_level. Activations are N(0, 1), codes and zero points uniform, scales |N(0, 0.02)|, biases
N(0, 0.1): the distributions of the benchmark's configurations.
"""

import math

import numpy as np
import torch

from onnx_light_cpu_b200 import MatMulNBitsSession, MatMulNBitsWeights, register_kernels
from onnx_light_cpu_b200.tools.decoder_layer import STAGES, DecoderLayerProjections

DEVICE = "cuda:0"

register_kernels()  # once per process, before an evaluator builds its sessions


def _node(name, m, k, n, bits, block, zp, bias, level, kind="node"):
    return {"name": name, "kind": kind, "m": m, "k": k, "n": n, "bits": bits, "block": block, "zp": zp, "bias": bias,
            "level": level}


def _layer(name, m, hidden, kv, ffn, bits, block, zp, level):
    return {"name": name, "kind": "layer", "m": m, "hidden": hidden, "kv": kv, "ffn": ffn, "bits": bits, "block": block,
            "zp": zp, "bias": False, "level": level}


def listed():
    return [
        # one token through one square node: the smallest call, all latency
        _node("decode_node_m1", 1, 4096, 4096, 4, 32, False, False, 0),
        # one token through the evaluator's operator: host array in, host array out, every call waits
        _node("decode_operator_m1", 1, 4096, 14336, 4, 128, True, True, 0, kind="operator"),
        # one sequence being generated: a decoder layer's projections at one token
        _layer("decode_layer_m1", 1, 4096, 1024, 14336, 4, 32, False, 0),
        # sixteen sequences generated together, activations kept at full precision
        _layer("decode_layer_m16", 16, 4096, 1024, 14336, 4, 32, False, 0),
        # the same layer of a model that was exported for int8 activations
        _layer("decode_layer_m16_level4", 16, 4096, 1024, 14336, 4, 32, False, 4),
        # four sequences (or a four-token draft being verified), coarse blocks, all optional operands
        _node("decode_node_m4", 4, 4096, 14336, 4, 128, True, True, 0),
        # the output projection of the next token, unsharded: the largest weight stream
        _node("lm_head_m1", 1, 4096, 128256, 4, 32, True, False, 0),
        # the same for eight sequences with the 8-bit weights that exporters give this layer
        _node("lm_head_m8_8bit", 8, 4096, 128256, 8, 32, True, False, 0),
        # a short prompt on sizes that are no power of two, an odd number of columns
        _node("short_prompt_ragged", 45, 5760, 9001, 4, 64, True, True, 0),
        # the prompt of a model that was exported for int8 activations
        _node("prefill_m512_level4", 512, 4096, 4096, 4, 32, False, False, 4),
        # an ordinary prompt
        _node("prefill_m2048", 2048, 4096, 4096, 4, 64, True, False, 0),
        # a long prompt, or several batched: the largest call
        _node("prefill_m8192", 8192, 4096, 4096, 4, 64, True, False, 0),
    ]


MOST_FLOPS = 2 * 8192 * 4096 * 4096
MOST_BYTES = 600e6


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _multiple(value, of):
    return max(of, (value + of // 2) // of * of)


def draw(rng):
    """One more case: any token count up to a long prompt, rows of 1024 to 14336 codes (whole blocks, multiples of 64),
    any number of columns, every block size, both code widths and both levels."""
    kind = rng.choice(["node"] * 7 + ["layer"] * 2 + ["operator"])
    bits = rng.choice([4, 4, 4, 8])
    block = rng.choice([16] + [32] * 8 + [64] * 4 + [128] * 6 + [256])
    level = rng.choice([0, 0, 4])
    step = max(64, block)
    while True:
        if kind == "layer":
            hidden = _multiple(_log(rng, 1024, 5120), step)
            case = _layer("", _log(rng, 1, 48), hidden, _multiple(hidden // rng.choice([1, 2, 4, 8]), 64),
                          _multiple(int(hidden * rng.uniform(2.5, 4.0)), step), bits, block, rng.random() < 0.5, level)
        else:
            k = _multiple(_log(rng, 1024, 14336), step)
            # mostly projections, sometimes a vocabulary
            n = _log(rng, 16384, 131072) if rng.random() < 0.1 else _log(rng, 512, 14336)
            if rng.random() < 0.7:
                n = _multiple(n, 64)
            m = _log(rng, 1, 8192 if kind == "node" else 512)
            m = max(1, min(m, MOST_FLOPS // (2 * k * n)))
            case = _node("", m, k, n, bits, block, rng.random() < 0.6, rng.random() < 0.3, level, kind=kind)
        del case["name"]
        cost = work(case)
        if cost["bytes"] <= MOST_BYTES and cost["flops"] <= MOST_FLOPS:
            return case


def _shapes(case):
    """Name, K and N of the case's nodes."""
    if case["kind"] != "layer":
        return [("node", case["k"], case["n"])]
    h, kv, f = case["hidden"], case["kv"], case["ffn"]
    return [("q", h, h), ("k", h, kv), ("v", h, kv), ("o", h, h), ("gate", h, f), ("up", h, f), ("down", f, h)]


def work(case):
    """Packed codes, scales, zero points and bias of every node, each different activation and each result once."""
    m, bits, block = case["m"], case["bits"], case["block"]
    total, flops = 0, 0
    for _, k, n in _shapes(case):
        blocks = -(-k // block)
        total += n * blocks * (block * bits // 8) + 4 * n * blocks + 4 * m * n
        total += n * ((blocks * bits + 7) // 8) if case["zp"] else 0
        total += 4 * n if case["bias"] else 0
        flops += 2 * m * k * n
    if case["kind"] == "layer":
        total += 4 * m * (3 * case["hidden"] + case["ffn"])
    else:
        total += 4 * m * case["k"]
    return {"bytes": total, "flops": flops}


def tolerance(case):
    """Four times what was measured against the same product in 64 bits: a few 1e-7 for 32-bit sums (up to sixteen tokens, and
    int8 activations at any number), 3e-3 with bf16 operands (more tokens at level 0)."""
    if case["m"] > 16 and case["level"] == 0:
        return {"rel": 1.2e-2}
    return {"rel": 3e-6}


class _Operands:
    """Constant operands of one node as CUDA tensors (the fields DecoderLayerProjections reads)."""

    def __init__(self, case, k, n, gen):
        bits, block = case["bits"], case["block"]
        blocks = -(-k // block)
        self.k, self.n, self.bits, self.block_size = k, n, bits, block
        self.b = torch.randint(0, 256, (n, blocks, block * bits // 8), dtype=torch.uint8, device=DEVICE, generator=gen)
        self.scales = torch.randn(n * blocks, device=DEVICE, generator=gen).abs_().mul_(0.02)
        self.zero_points = self.bias = None
        if case["zp"]:
            self.zero_points = torch.randint(0, 256, (n, (blocks * bits + 7) // 8), dtype=torch.uint8, device=DEVICE,
                                             generator=gen)
        if case["bias"]:
            self.bias = torch.randn(n, device=DEVICE, generator=gen).mul_(0.1)


def _host(tensor):
    return None if tensor is None else tensor.cpu().numpy()


def _drawn(case, seed):
    """Operands by node, activations by stage."""
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    operands = {name: _Operands(case, k, n, gen) for name, k, n in _shapes(case)}
    stages = STAGES if case["kind"] == "layer" else (("node", ("node",)),)
    inputs = {stage: torch.randn(case["m"], operands[names[0]].k, device=DEVICE, generator=gen) for stage, names in stages}
    return operands, inputs


def prepare(case, seed):
    m, kind = case["m"], case["kind"]
    operands, inputs = _drawn(case, seed)
    torch.cuda.synchronize()  # the weights are in place before a handle lays out what it derives from them
    if kind == "layer":
        layer = DecoderLayerProjections(operands)
        layer.outputs(m)
        return {"case": case, "layer": layer, "inputs": inputs}
    node, a = operands["node"], inputs["node"]
    options = {"K": node.k, "N": node.n, "bits": node.bits, "block_size": node.block_size}
    if kind == "operator":
        session = MatMulNBitsSession(_host(node.b), _host(node.scales), _host(node.zero_points), _host(node.bias),
                                     accuracy_level=case["level"], **options)
        return {"case": case, "session": session, "a": _host(a)}
    weights = MatMulNBitsWeights(node.b, node.scales, node.zero_points, node.bias, **options)
    return {"case": case, "weights": weights, "a": a, "y": torch.empty(m, node.n, device=DEVICE)}


def run(state):
    case = state["case"]
    if case["kind"] == "layer":
        return state["layer"].run(state["inputs"], accuracy_level=case["level"])
    if case["kind"] == "operator":
        return state["session"].run(state["a"])
    state["weights"].matmul_device(state["a"], state["y"], accuracy_level=case["level"])
    return state["y"]


def _product64(case, operand, a):
    """Y of one node in 64 bits. At level 4 the activations are first the operator's int8 codes, one scale per block."""
    m, k, n, bits, block = case["m"], operand.k, operand.n, operand.bits, operand.block_size
    blocks = k // block
    if case["level"] == 4:
        groups = a.cpu().numpy().reshape(m, blocks, block)  # on the host: the codes follow from IEEE single divisions
        scale = np.abs(groups).max(axis=2, keepdims=True) / np.float32(127.0)
        codes = np.rint(groups / scale).clip(-127.0, 127.0)
        a = torch.from_numpy(codes.astype(np.float64) * scale.astype(np.float64)).to(DEVICE).reshape(m, k)
    a = a.double()
    y = torch.empty(m, n, dtype=torch.float64, device=DEVICE)
    rows = max(1, (1 << 27) // k)  # columns of Y at a time: about 1 GB of weights in 64 bits
    for first in range(0, n, rows):
        codes = operand.b[first:first + rows].flatten(1)
        if bits == 4:
            codes = torch.stack((codes & 15, codes >> 4), dim=2)
        codes = codes.reshape(-1, blocks, block).double()
        zero = torch.full((codes.shape[0], blocks), float(1 << (bits - 1)), dtype=torch.float64, device=DEVICE)
        if operand.zero_points is not None:
            zero = operand.zero_points[first:first + rows]
            if bits == 4:
                zero = torch.stack((zero & 15, zero >> 4), dim=2).flatten(1)[:, :blocks]
            zero = zero.double()
        scale = operand.scales.view(n, blocks)[first:first + rows].double()
        y[:, first:first + rows] = a @ ((codes - zero[:, :, None]) * scale[:, :, None]).flatten(1).t()
    if operand.bias is not None:
        y += operand.bias.double()
    return y


def exact(case, seed):
    operands, inputs = _drawn(case, seed)
    if case["kind"] == "layer":
        return {name: _product64(case, operands[name], inputs[stage]) for stage, names in STAGES for name in names}
    return _product64(case, operands["node"], inputs["node"])
