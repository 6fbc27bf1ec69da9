"""What the framework's users have it do, as cases that can be timed: training steps of LUT networks (dense, convolutional, on
fp32 frames in probability and in binary mode, on bit frames, on modulated frames) and inference of frozen networks on bit frames
(on the device, from host buffers, through the C++ host classes), each through the public entry points and over the range of sizes
from one small batch to layers that fill the GPU.

listed() names twelve cases, draw() gives further ones of the same ranges, prepare() makes what a program has in hand before the
call, run() is one pass, work() what a pass cannot do without, tolerance() how far two correct implementations may be apart.
"""
import math

import numpy as np
import torch

from binarybrain_b200 import conv, ops
from binarybrain_b200 import core
from binarybrain_b200.dist import ShardedDifferentiableLut6

MODULATION = 7                       # bit frames per fp32 frame of the modulated network
FILTER = 3                           # 3 x 3 "same" convolutions, 2 x 2 pooling
BLOCKS = ((216, 36, 32), (216, 36, 32)), ((384, 64), (384, 64))          # per-pixel layer widths of the two convolution blocks
HEAD = (1024, 420, 70, 10)           # dense head of the convolutional network

# work of one LUT evaluation on fp32 inputs: 63 multiply-adds forward; backward the evaluation again, the reverse walk of its 63 nodes
# and the 64 table-gradient sums
FLOPS_FORWARD, FLOPS_BACKWARD = 126.0, 379.0


def listed():
    return [
        # the small MLP on 784 features, one optimizer step on a batch of 512: launches and host work count here
        {"name": "mlp_step_512", "kind": "mlp_step", "n0": 784, "n1": 1024, "n2": 420, "n3": 70, "frames": 512, "binary": False},
        # the same kind of network in the layers' default (binary) mode on a small batch that is no multiple of a row or a warp
        {"name": "mlp_step_binary_100", "kind": "mlp_step", "n0": 784, "n1": 360, "n2": 240, "n3": 60, "frames": 100, "binary": True},
        # the wide regression network on one GPU's share of a batch: 65536-node layers, fresh tables
        {"name": "stack_65536x4096", "kind": "stack", "nodes": 65536, "layers": 2, "frames": 4096, "binary": False, "table_sd": 0.01},
        # an ordinary stack with sizes that divide nothing
        {"name": "stack_3000x5001", "kind": "stack", "nodes": 3000, "layers": 3, "frames": 5001, "binary": False, "table_sd": 0.25},
        # a stack in binary mode on fp32 frames
        {"name": "stack_binary_8192x16384", "kind": "stack", "nodes": 8192, "layers": 2, "frames": 16384, "binary": True, "table_sd": 0.25},
        # bit-packed frames in and between the layers, fp32 gradients
        {"name": "bit_stack_8192x16384", "kind": "bit_stack", "nodes": 8192, "layers": 2, "frames": 16384},
        # binary modulation: 3 x 32 x 32 images, seven bit frames per image, two stochastic layers, demodulation to ten outputs
        {"name": "modulated_256", "kind": "modulated", "side": 32, "n1": 4096, "n2": 1020, "frames": 256},
        # the LUT-CNN training step (3 x 3 lowering, per-pixel trees, pooling, dense head) on 256 images
        {"name": "cnn_step_256", "kind": "cnn_step", "side": 32, "frames": 256},
        # the frozen LUT-CNN on bit frames
        {"name": "cnn_bits_1024", "kind": "cnn_bits", "side": 32, "frames": 1024},
        # one frozen layer at the largest size: 2^20 bit frames
        {"name": "bits_16384x1048576", "kind": "bits", "nodes": 16384, "layers": 1, "frames": 1 << 20},
        # a small frozen network through the C++ host classes, one batch of 200 frames: the smallest call
        {"name": "bits_classes_200", "kind": "bits_classes", "n0": 784, "n1": 1024, "n2": 420, "n3": 70, "frames": 200},
        # host buffers in, host buffers out, ragged sizes
        {"name": "bits_host_5000x100003", "kind": "bits_host", "nodes": 5000, "frames": 100003},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, even over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _area(rng, nodes_lo, nodes_hi, frames_lo, frames_hi, most):
    """(nodes, frames) of a layer with at most `most` node-frames."""
    nodes = _log(rng, nodes_lo, nodes_hi)
    return nodes, _log(rng, frames_lo, max(frames_lo, min(frames_hi, most // nodes)))


def draw(rng):
    kind = rng.choice(["mlp_step", "mlp_step", "stack", "stack", "stack", "bit_stack", "modulated", "cnn_step", "cnn_bits", "bits", "bits",
                       "bits_classes", "bits_host"])
    if kind == "mlp_step":
        return {"kind": kind, "n0": _log(rng, 64, 3072), "n1": _log(rng, 128, 4096), "n2": _log(rng, 64, 1024), "n3": 10 * _log(rng, 2, 24),
                "frames": _log(rng, 16, 4096), "binary": rng.random() < 0.5}
    if kind == "stack":
        nodes, frames = _area(rng, 1024, 65536, 256, 32768, 1 << 27)
        return {"kind": kind, "nodes": nodes, "layers": rng.choice([1, 2, 3]), "frames": frames, "binary": rng.random() < 0.4,
                "table_sd": rng.choice([0.01, 0.25])}
    if kind == "bit_stack":
        nodes, frames = _area(rng, 1024, 32768, 256, 32768, 1 << 27)
        return {"kind": kind, "nodes": nodes, "layers": rng.choice([1, 2, 3]), "frames": frames}
    if kind == "modulated":
        return {"kind": kind, "side": rng.randint(16, 32), "n1": _log(rng, 1024, 8192), "n2": 10 * _log(rng, 10, 200), "frames": _log(rng, 16, 1024)}
    if kind == "cnn_step":
        return {"kind": kind, "side": rng.randint(16, 32), "frames": _log(rng, 8, 256)}
    if kind == "cnn_bits":
        return {"kind": kind, "side": rng.randint(16, 32), "frames": _log(rng, 32, 2048)}
    if kind == "bits":
        nodes, frames = _area(rng, 256, 32768, 256, 1 << 20, 1 << 33)
        return {"kind": kind, "nodes": nodes, "layers": rng.choice([1, 2, 3]), "frames": frames}
    if kind == "bits_classes":
        return {"kind": kind, "n0": _log(rng, 64, 3072), "n1": _log(rng, 128, 4096), "n2": _log(rng, 64, 1024), "n3": 10 * _log(rng, 2, 24),
                "frames": _log(rng, 1, 65536)}
    nodes, frames = _area(rng, 256, 16384, 256, 1 << 18, 1 << 30)
    return {"kind": kind, "nodes": nodes, "frames": frames}


# ------------------------------------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _wiring(n_in, n_out, g):
    """Six distinct random inputs per node."""
    if n_in * n_out <= 1 << 22:
        return torch.rand((n_out, n_in), device="cuda", generator=g).argsort(dim=1)[:, :6].to(torch.int32).contiguous()
    idx = torch.randint(0, n_in, (n_out, 6), device="cuda", generator=g)
    for _ in range(4):                                          # re-draw the few nodes with a repeat
        s = idx.sort(dim=1).values
        bad = (s[:, 1:] == s[:, :-1]).any(dim=1, keepdim=True)
        idx = torch.where(bad, torch.randint(0, n_in, (n_out, 6), device="cuda", generator=g), idx)
    return idx.to(torch.int32).contiguous()


def _tables(nodes, sd, g):
    return (torch.randn((nodes, 64), device="cuda", generator=g) * sd + 0.5).clamp_(0, 1)


def _frames(nodes, frames, g):
    """fp32 frames uniform in [0, 1), rows padded as the framework pads them."""
    x = torch.rand((nodes, ops.fp32_stride(frames)), device="cuda", generator=g)
    x[:, frames:] = 0
    return x


def _bits(nodes, frames, g):
    """Bernoulli(1/2) bit frames; the bits past the last frame are clear."""
    x = torch.randint(-2**31, 2**31 - 1, (nodes, ops.bit_stride(frames)), dtype=torch.int32, device="cuda", generator=g)
    words = (frames + 31) // 32
    x[:, words:] = 0
    if frames % 32:
        x[:, words - 1] &= (1 << frames % 32) - 1
    return x


def _truth_tables(nodes, g):
    return torch.randint(-2**31, 2**31 - 1, (nodes, 2), dtype=torch.int32, device="cuda", generator=g)


def _layer(n_in, n_out, sd, binary, g):
    return ShardedDifferentiableLut6(_wiring(n_in, n_out, g), _tables(n_out, sd, g), n_in, binary=binary, sharded=False)


def _words(t, frames):
    """The words of bit frames that hold frames (the padding of a row is nobody's output)."""
    return t[:, :(frames + 31) // 32]


def prepare(case, seed):
    return _KINDS[case["kind"]][0](dict(case), _generator(seed), seed)


def run(state):
    return _KINDS[state["kind"]][1](state)


def work(case):
    return _KINDS[case["kind"]][2](case)


def tolerance(case):
    """Inference on bit frames is exact.  fp32 training sums in fp32 over frames and consumers in no fixed order; batch norm multiplies
    the rounding of a LUT value near 1/2 by gamma * rstd (up to 95 on fresh tables), once per layer on the way back."""
    kind = case["kind"]
    if kind in ("cnn_bits", "bits", "bits_classes", "bits_host"):
        return "exact"
    if kind == "modulated":
        return {"rel": 1e-5}
    return {"rel": 1e-4, "max": 1e-2}


# ------------------------------------------------------------------------------------------------ small MLP: a whole optimizer step
def _prepare_mlp(s, g, seed):
    widths, F = [s["n0"], s["n1"], s["n2"], s["n3"]], s["frames"]
    s["x"] = _frames(widths[0], F, g)
    labels = torch.randint(0, 10, (F,), device="cuda", generator=g)
    s["t"] = torch.zeros((10, ops.fp32_stride(F)), device="cuda")
    s["t"][labels, torch.arange(F, device="cuda")] = 1.0
    s["layers"] = [_layer(a, b, 0.25, s["binary"], g) for a, b in zip(widths, widths[1:])]
    s["opt"] = ops.Adam([l.W for l in s["layers"]], [l.dW for l in s["layers"]])
    return s


def _run_mlp(s):
    F, h = s["frames"], s["x"]
    for l in s["layers"]:
        ops.clamp_(l.W)
        h = l.forward(h, F, F)
    scores = ops.reduce_forward(h, 10, F)
    dy, loss = ops.softmax_cross_entropy(scores, s["t"], F)
    dy = ops.reduce_backward(dy, h.shape[0], F)
    for l in reversed(s["layers"]):
        dy = l.backward(dy)
    s["opt"].update()
    return {"loss": loss, "scores": scores[:, :F], "dx": dy[:, :F], "W": [l.W for l in s["layers"]], "mean": [l.running_mean for l in s["layers"]],
            "var": [l.running_var for l in s["layers"]]}


def _work_mlp(c):
    widths, F = [c["n0"], c["n1"], c["n2"], c["n3"]], c["frames"]
    nodes = sum(widths[1:])
    # x read in both passes, y written and read again by the backward pass, dy read, dx written; W, m and v read and written
    byt = sum(8.0 * a * F + 12.0 * b * F for a, b in zip(widths, widths[1:])) + 4.0 * widths[0] * F + nodes * 64 * 4 * 6
    return {"bytes": byt, "flops": 0.0 if c["binary"] else nodes * F * (FLOPS_FORWARD + FLOPS_BACKWARD)}


# ------------------------------------------------------------------------------------------------ stack of equal layers: loss and all gradients
def _prepare_stack(s, g, seed):
    n, F = s["nodes"], s["frames"]
    s["x"], s["t"] = _frames(n, F, g), _frames(n, F, g)
    s["layers"] = [_layer(n, n, s["table_sd"], s["binary"], g) for _ in range(s["layers"])]
    s["y"] = [torch.empty_like(s["x"]) for _ in s["layers"]]
    s["g"] = [torch.empty_like(s["x"]) for _ in range(2)]
    return s


def _run_stack(s):
    F, h = s["frames"], s["x"]
    for l in s["layers"]:
        l.dW.zero_()
    for l, y in zip(s["layers"], s["y"]):
        h = l.forward(h, F, F, y=y)
    dy, loss = ops.mean_squared_error(h, s["t"], F, dy=s["g"][0])
    for k, l in enumerate(reversed(s["layers"])):
        dy = l.backward(dy, dx=s["g"][(k + 1) % 2])
    return {"loss": loss.sum(), "y": h[:, :F], "dx": dy[:, :F], "dW": [l.dW for l in s["layers"]], "mean": [l.running_mean for l in s["layers"]],
            "var": [l.running_var for l in s["layers"]]}


def _work_stack(c):
    nf = float(c["nodes"]) * c["frames"]
    # per layer x read and y written, then x and dy read and dx written; the loss reads y and the target and writes dy
    return {"bytes": nf * (20.0 * c["layers"] + 12.0), "flops": 0.0 if c["binary"] else nf * c["layers"] * (FLOPS_FORWARD + FLOPS_BACKWARD)}


# ------------------------------------------------------------------------------------------------ the same on bit frames
def _prepare_bit_stack(s, g, seed):
    n, F = s["nodes"], s["frames"]
    s["x"], s["dy"] = _bits(n, F, g), torch.randn((n, ops.fp32_stride(F)), device="cuda", generator=g) / F
    s["layers"] = [{"idx": _wiring(n, n, g), "W": _tables(n, 0.25, g), "dW": torch.zeros((n, 64), device="cuda"), "rm": torch.zeros(n, device="cuda"),
                    "rv": torch.ones(n, device="cuda"), "y": torch.zeros_like(s["x"])} for _ in range(s["layers"])]
    s["g"] = [torch.empty_like(s["dy"]) for _ in range(2)]
    return s


def _run_bit_stack(s):
    n, F, h, saved = s["nodes"], s["frames"], s["x"], []
    for l in s["layers"]:
        l["dW"].zero_()
    for l in s["layers"]:
        y, mean, rstd = ops.differentiable_lut6_forward_training(h, l["idx"], l["W"], l["rm"], l["rv"], F, y=l["y"])
        saved.append((h, mean, rstd))
        h = y
    dy = s["dy"]
    for k, (l, (x, mean, rstd)) in enumerate(zip(reversed(s["layers"]), reversed(saved))):
        dy = ops.differentiable_lut6_backward(x, dy, l["idx"], l["W"], l["dW"], mean, rstd, n, F, dx=s["g"][k % 2])
    return {"y": _words(h, F), "dx": dy[:, :F], "dW": [l["dW"] for l in s["layers"]], "mean": [l["rm"] for l in s["layers"]],
            "var": [l["rv"] for l in s["layers"]]}


def _work_bit_stack(c):
    # per layer the bits of x and y forward, the bits of x, dy and dx backward
    return {"bytes": float(c["nodes"]) * c["frames"] * c["layers"] * (8.0 + 3.0 / 8.0), "flops": 0.0}


# ------------------------------------------------------------------------------------------------ modulated network, forward and backward
def _prepare_modulated(s, g, seed):
    n0, B = 3 * s["side"] ** 2, s["frames"]
    s["x"], s["th"] = _frames(n0, B, g), _frames(n0, B * MODULATION, g)
    s["idx"] = [_wiring(n0, s["n1"], g), _wiring(s["n1"], s["n2"], g)]
    s["W"] = [_tables(s["n1"], 0.01, g), _tables(s["n2"], 0.01, g)]
    s["dW"] = [torch.zeros_like(w) for w in s["W"]]
    s["dy"] = torch.randn((10, ops.fp32_stride(B)), device="cuda", generator=g) / B
    return s


def _run_modulated(s):
    n0, n1, n2, B, F = 3 * s["side"] ** 2, s["n1"], s["n2"], s["frames"], s["frames"] * MODULATION
    for w in s["dW"]:
        w.zero_()
    xb = ops.real_to_binary(s["x"], B, frame_mod=MODULATION, thresholds=s["th"])
    h1 = ops.stochastic_lut6_forward(xb, s["idx"][0], s["W"][0], F)
    h2 = ops.stochastic_lut6_forward(h1, s["idx"][1], s["W"][1], F)
    y = ops.binary_to_real(h2, n2, 10, B, frame_mux=MODULATION)
    g = ops.binary_to_real_backward(s["dy"], n2, B, frame_mux=MODULATION)
    g = ops.stochastic_lut6_backward(h1, g, s["idx"][1], s["W"][1], s["dW"][1], n1, F)
    dx = ops.stochastic_lut6_backward(xb, g, s["idx"][0], s["W"][0], s["dW"][0], n0, F)
    return {"bits": _words(xb, F), "h": h2[:, :F], "y": y[:, :B], "dx": dx[:, :F], "dW": s["dW"]}


def _work_modulated(c):
    n0, n1, n2, B, F = 3.0 * c["side"] ** 2, c["n1"], c["n2"], c["frames"], c["frames"] * MODULATION
    # images and thresholds in, bits out; bits in, h1 out; h1 in, h2 out and in; then h1 and the two gradients, the bits and the last one
    byt = n0 * (4.0 * B + 4.0 * F + F / 8.0) + n0 * F / 8.0 + n1 * F * 8.0 + n2 * F * 8.0 + n2 * F * 8.0 + n1 * F * 12.0 + n0 * F * (4.0 + 1.0 / 8.0)
    return {"bytes": byt, "flops": n2 * F * (FLOPS_FORWARD + FLOPS_BACKWARD)}


# ------------------------------------------------------------------------------------------------ LUT-CNN
def _shapes(side):
    """((channels, side, widths) of every convolution block, nodes of the dense head's input)."""
    c, blocks = 3, []
    for convs in BLOCKS:
        block = []
        for widths in convs:
            block.append((c, side, widths))
            c = widths[-1]
        blocks.append(block)
        side = (side + 1) // 2
    return blocks, c * side * side


def _prepare_cnn(s, g, seed):
    blocks, dense_in = _shapes(s["side"])
    layers = []
    for block in blocks:
        for c, side, widths in block:
            fan = [c * FILTER * FILTER] + list(widths)
            inner = [_layer(a, b, 0.25, False, g) for a, b in zip(fan, fan[1:])]
            layers.append(conv.Convolution2d(inner, c, side, side, FILTER, FILTER, padding="same"))
        layers.append(conv.MaxPooling(block[-1][2][-1], side, side, 2, 2))
    fan = [dense_in] + list(HEAD)
    s["net"] = conv.Sequential(layers + [_layer(a, b, 0.25, False, g) for a, b in zip(fan, fan[1:])])
    s["x"] = _frames(3 * s["side"] ** 2, s["frames"], g)
    s["dy"] = torch.randn((HEAD[-1], ops.fp32_stride(s["frames"])), device="cuda", generator=g) / s["frames"]
    return s


def _run_cnn(s):
    luts = s["net"].lut_layers()
    for l in luts:
        l.dW.zero_()
    y = s["net"].forward(s["x"], s["frames"])
    dx = s["net"].backward(s["dy"])
    return {"y": y[:, :s["frames"]], "dx": dx[:, :s["frames"]], "dW": [l.dW for l in luts], "mean": [l.running_mean for l in luts]}


def _work_cnn(c):
    B, byt, nf = c["frames"], 0.0, 0.0
    blocks, dense_in = _shapes(c["side"])
    for block in blocks:
        for ch, side, widths in block:
            P = side * side
            fan = [ch] + list(widths)                            # the 3 x 3 neighbourhoods need not be written out
            byt += sum(8.0 * a + 8.0 * b for a, b in zip(fan, fan[1:])) * P * B + 4.0 * fan[0] * P * B
            nf += float(sum(widths)) * P * B
        byt += block[-1][2][-1] * block[-1][1] ** 2 * B * 10.0    # pooling: image in and a quarter out, both ways
    fan = [dense_in] + list(HEAD)
    byt += sum(12.0 * a + 8.0 * b for a, b in zip(fan, fan[1:])) * B
    nf += float(sum(HEAD)) * B
    return {"bytes": byt, "flops": nf * (FLOPS_FORWARD + FLOPS_BACKWARD)}


def _prepare_cnn_bits(s, g, seed):
    blocks, dense_in = _shapes(s["side"])

    def chain(fan):
        return [(_wiring(a, b, g), _truth_tables(b, g)) for a, b in zip(fan, fan[1:])]

    s["blocks"] = [[(c, side, chain([c * FILTER * FILTER] + list(widths))) for c, side, widths in block] for block in blocks]
    s["head"] = chain([dense_in] + list(HEAD))
    s["x"] = _bits(3 * s["side"] ** 2, s["frames"], g)
    return s


def _run_cnn_bits(s):
    F, h = s["frames"], s["x"]
    for block in s["blocks"]:
        for c, side, layers in block:
            h = ops.im2col_forward(h, F, c, side, side, FILTER, FILTER, padding="same")
            for idx, table in layers:
                h = ops.binary_lut6_forward(h, idx, table, F * side * side)
            h = ops.col2im_forward(h, h.shape[0], side, side, F)
        h = ops.maxpool_forward(h, F, h.shape[0] // (side * side), side, side, 2, 2)
    for idx, table in s["head"]:
        h = ops.binary_lut6_forward(h, idx, table, F)
    return _words(h, F)


def _work_cnn_bits(c):
    B, blocks, dense_in = c["frames"], *_shapes(c["side"])
    bits = 0.0
    for block in blocks:
        for ch, side, widths in block:
            fan = [ch] + list(widths)
            bits += sum(a + b for a, b in zip(fan, fan[1:])) * side * side * B
        bits += block[-1][2][-1] * block[-1][1] ** 2 * B * 1.25
    fan = [dense_in] + list(HEAD)
    bits += sum(a + b for a, b in zip(fan, fan[1:])) * B
    return {"bytes": bits / 8.0, "flops": 0.0}


# ------------------------------------------------------------------------------------------------ frozen layers on bit frames
def _prepare_bits(s, g, seed):
    n, F = s["nodes"], s["frames"]
    s["x"] = _bits(n, F, g)
    s["layers"] = [(_wiring(n, n, g), _truth_tables(n, g)) for _ in range(s["layers"])]
    s["y"] = [torch.zeros_like(s["x"]) for _ in s["layers"]]
    return s


def _run_bits(s):
    h = s["x"]
    for (idx, table), y in zip(s["layers"], s["y"]):
        h = ops.binary_lut6_forward(h, idx, table, s["frames"], y=y)
    return _words(h, s["frames"])


def _work_bits(c):
    return {"bytes": c["layers"] * (c["nodes"] * 2.0 * c["frames"] / 8.0 + 32.0 * c["nodes"]), "flops": 0.0}


class _DeviceView:
    """The device memory of a frame buffer for torch.as_tensor, which keeps this object, and with it the buffer, alive."""

    def __init__(self, buffer):
        self._buffer = buffer
        stride = buffer.get_frame_stride()
        words = (buffer.get_frame_size() + 31) // 32
        self.__cuda_array_interface__ = {"data": (buffer.lock_device(), False), "shape": (buffer.get_node_size(), words), "strides": (stride, 4),
                                         "typestr": "<i4", "version": 3}


def _prepare_classes(s, g, seed):
    s["net"] = core.Sequential.create()
    for k, n in enumerate((s["n1"], s["n2"], s["n3"])):
        s["net"].add(core.BinaryLut6_bit_fp32.create([n], seed=16 * seed + k + 1))
    s["net"].set_input_shape([s["n0"]])
    s["x"] = core.FrameBuffer.from_numpy_fp32(np.random.default_rng(seed).integers(0, 2, (s["frames"], s["n0"])).astype(np.float32), core.TYPE_BIT)
    s["x"].lock_device()                                        # the batch is on the device
    return s


def _run_classes(s):
    return torch.as_tensor(_DeviceView(s["net"].forward(s["x"], False)), device="cuda")


def _work_classes(c):
    widths = [c["n0"], c["n1"], c["n2"], c["n3"]]
    return {"bytes": sum((a + b) * c["frames"] / 8.0 + 32.0 * b for a, b in zip(widths, widths[1:])), "flops": 0.0}


def _prepare_host(s, g, seed):
    n, F = s["nodes"], s["frames"]
    s["x"] = _bits(n, F, g).cpu().pin_memory()
    s["y"] = torch.zeros_like(s["x"]).pin_memory()
    s["idx"], s["table"] = _wiring(n, n, g).cpu(), _truth_tables(n, g).cpu()
    return s


def _run_host(s):
    return _words(ops.binary_lut6_forward_host(s["x"], s["idx"], s["table"], s["frames"], y=s["y"]), s["frames"])


def _work_host(c):
    return {"bytes": c["nodes"] * 2.0 * c["frames"] / 8.0 + 32.0 * c["nodes"], "flops": 0.0}


_KINDS = {"mlp_step": (_prepare_mlp, _run_mlp, _work_mlp), "stack": (_prepare_stack, _run_stack, _work_stack),
          "bit_stack": (_prepare_bit_stack, _run_bit_stack, _work_bit_stack), "modulated": (_prepare_modulated, _run_modulated, _work_modulated),
          "cnn_step": (_prepare_cnn, _run_cnn, _work_cnn), "cnn_bits": (_prepare_cnn_bits, _run_cnn_bits, _work_cnn_bits),
          "bits": (_prepare_bits, _run_bits, _work_bits), "bits_classes": (_prepare_classes, _run_classes, _work_classes),
          "bits_host": (_prepare_host, _run_host, _work_host)}
