"""What users of this package have it do, as cases that can be timed and compared.

Five kinds of work, all through the public entry points of `oxionnx_b200.session` and with the
graphs of `oxionnx_b200.models` (the configurations of `bench.py`):

  mlp        the INT8 MLP                                       rows 1 .. 4096
  cnn_int8   the QLinearConv residual network                   batch 1 .. 1024
  cnn_f32    the float residual network                         batch 1 .. 64, TF32 or bf16 operands
  generator  the image-to-image float network with AdaIN heads  batch 1 .. 8
  encoder    the dynamic-INT8 transformer encoder               batch 1 .. 64, 16 .. 384 tokens
  node       a residual block dispatched one node at a time, the way a host engine hands single
             nodes to the provider, with the values between the nodes resident on the device

and three ways in:

  device     inputs and outputs bound to the caller's device buffers (run_with_binding)
  host       numpy feeds in, numpy results out (run)
  stream     several batches from page-locked memory with two in flight (run_pipelined)

A program plans a session once and then feeds it one request after the other, so the states of one
case share their session and differ in the inputs; only the most recent session is kept alive here,
and it goes when the last state that uses it does.
"""
import math
import weakref

import numpy as np
import torch

from oxionnx_b200 import models
from oxionnx_b200.graph import Node
from oxionnx_b200.session import CudaContext, Session, try_cuda_dispatch_resident

MLP_DIMS = (1024, 4096, 4096, 1024)
HIDDEN, HEADS, FFN, LAYERS, VOCAB = 768, 12, 3072, 12, 30522
STREAM_BATCHES = 4


def listed():
    return [
        # one row from a host program that waits for its answer: nothing but latency
        {"name": "mlp one row", "kind": "mlp", "rows": 1, "spelling": "qlinearconv", "io": "host"},
        # the benchmark's configuration of the MLP
        {"name": "mlp 64 rows", "kind": "mlp", "rows": 64, "spelling": "qlinearconv", "io": "device"},
        # scoring a table in chunks, the last of them ragged; per-tensor scales
        {"name": "mlp 1500 rows", "kind": "mlp", "rows": 1500, "spelling": "qlinearmatmul", "io": "device"},
        # a host engine that owns the graph and gives the provider single nodes
        {"name": "node block", "kind": "node", "batch": 2, "channels": 64, "height": 28, "width": 28},
        # one camera frame, already quantised, through a recorded graph
        {"name": "cnn int8 one frame", "kind": "cnn_int8", "batch": 1, "image": 224, "io": "host", "typed": True, "graph": True},
        # a queue of f32 frames on the host, batched as they come
        {"name": "cnn int8 stream of 37", "kind": "cnn_int8", "batch": 37, "image": 224, "io": "stream", "typed": False, "graph": True},
        # the benchmark's headline configuration
        {"name": "cnn int8 1024", "kind": "cnn_int8", "batch": 1024, "image": 224, "io": "device", "typed": False, "graph": True},
        # one frame on the device, float network
        {"name": "cnn f32 one frame", "kind": "cnn_f32", "batch": 1, "image": 224, "io": "device", "precision": "tf32", "graph": True},
        # the benchmark's configuration of the float network
        {"name": "cnn f32 32", "kind": "cnn_f32", "batch": 32, "image": 224, "io": "device", "precision": "tf32", "graph": True},
        # a few faces of a video at once
        {"name": "generator 4", "kind": "generator", "batch": 4, "io": "device", "graph": True},
        # a couple of short, ragged sentences
        {"name": "encoder 2x77", "kind": "encoder", "batch": 2, "seq": 77, "io": "device", "graph": True},
        # the benchmark's configuration of the encoder
        {"name": "encoder 64x128", "kind": "encoder", "batch": 64, "seq": 128, "io": "device", "graph": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mlp", "cnn_int8", "cnn_f32", "generator", "encoder", "encoder", "node"])
    graph = rng.random() < 0.7
    if kind == "mlp":
        return {"kind": kind, "rows": _log_int(rng, 1, 4096), "spelling": rng.choice(["qlinearconv", "qlinearmatmul"]), "io": rng.choice(["device", "host"])}
    if kind == "cnn_int8":
        io = rng.choice(["device", "device", "host", "stream"])
        return {"kind": kind, "batch": _log_int(rng, 1, 512 if io == "device" else 96), "image": rng.choice([160, 192, 224, 224, 256]), "io": io,
                "typed": rng.random() < 0.5, "graph": graph}
    if kind == "cnn_f32":
        return {"kind": kind, "batch": _log_int(rng, 1, 64), "image": rng.choice([160, 192, 224, 224, 256]), "io": rng.choice(["device", "device", "host"]),
                "precision": rng.choice(["tf32", "bf16"]), "graph": graph}
    if kind == "generator":
        return {"kind": kind, "batch": _log_int(rng, 1, 8), "io": rng.choice(["device", "host"]), "graph": graph}
    if kind == "encoder":
        seq = _log_int(rng, 16, 384)
        return {"kind": kind, "batch": _log_int(rng, 1, min(64, 8192 // seq)), "seq": seq, "io": rng.choice(["device", "device", "host"]), "graph": graph}
    return {"kind": kind, "batch": _log_int(rng, 1, 8), "channels": rng.choice([32, 64, 128, 256]), "height": _log_int(rng, 7, 56), "width": _log_int(rng, 7, 56)}


# ---- the layers of each network: (multiply-adds, weights) of one item ------------------------
def _convs(layers):
    return sum(o * o * cout * cin * k * k for cin, cout, k, o in layers), sum(cout * cin * k * k for cin, cout, k, o in layers)


def _cnn_layers(image):
    hw = (image - 1) // 2 + 1
    layers = [(3, 64, 7, hw)]
    hw = (hw - 1) // 2 + 1
    cin = 64
    for stage, blocks in enumerate((3, 4, 6, 3)):
        mid = 64 << stage
        for b in range(blocks):
            out = (hw - 1) // 2 + 1 if b == 0 and stage > 0 else hw
            layers += [(cin, mid, 1, hw), (mid, mid, 3, out), (mid, 4 * mid, 1, out)]
            if b == 0:
                layers.append((cin, 4 * mid, 1, out))
            cin, hw = 4 * mid, out
    return layers + [(cin, 1000, 1, 1)]


def _generator_layers():
    return ([(3, 128, 7, 128), (128, 256, 3, 128), (256, 512, 3, 64), (512, 1024, 3, 32)] + 12 * [(1024, 1024, 3, 32), (512, 2048, 1, 1)] +
            [(1024, 512, 3, 64), (512, 256, 3, 128), (256, 128, 3, 128), (128, 3, 7, 128)])


def _io_elements(case):
    """(input elements, output elements) of one batch."""
    kind = case["kind"]
    if kind == "mlp":
        return case["rows"] * MLP_DIMS[0], case["rows"] * MLP_DIMS[-1]
    b = case["batch"]
    if kind in ("cnn_int8", "cnn_f32"):
        return b * 3 * case["image"] ** 2, b * 1000
    if kind == "generator":
        return b * (3 * 128 * 128 + 512), b * 3 * 128 * 128
    if kind == "encoder":
        return 2 * b * case["seq"], b * case["seq"] * HIDDEN
    n = b * case["channels"] * case["height"] * case["width"]
    return n, n


def work(case):
    kind = case["kind"]
    n_in, n_out = _io_elements(case)
    if kind == "mlp":
        weights = sum(a * b for a, b in zip(MLP_DIMS, MLP_DIMS[1:]))
        return {"bytes": 4 * (n_in + n_out) + weights, "flops": 2 * case["rows"] * weights}
    b = case["batch"]
    if kind == "encoder":
        weights = LAYERS * (4 * HIDDEN * HIDDEN + 2 * HIDDEN * FFN)
        tokens = b * case["seq"]
        macs = tokens * weights + LAYERS * 2 * b * case["seq"] ** 2 * HIDDEN
        rows = min(tokens, VOCAB) + case["seq"]  # of the embedding tables
        return {"bytes": 4 * (n_in + n_out + rows * HIDDEN) + weights, "flops": 2 * macs}
    if kind == "node":
        c = case["channels"]
        macs, weights = 2 * n_in * c * 9, 2 * c * c * 9
        return {"bytes": 4 * (n_in + n_out + weights), "flops": 2 * macs}
    macs, weights = _convs(_generator_layers() if kind == "generator" else _cnn_layers(case["image"]))
    batches = STREAM_BATCHES if case["io"] == "stream" else 1
    lane = 1 if case.get("typed") else 4
    weight_lane = 1 if kind == "cnn_int8" else (2 if case.get("precision") == "bf16" else 4)
    return {"bytes": batches * (lane * n_in + 4 * n_out) + weight_lane * weights, "flops": 2 * macs * b * batches}


def tolerance(case):
    kind = case["kind"]
    if kind in ("mlp", "cnn_int8"):
        return "exact"  # integers all the way, and the last dequantisation is one multiplication
    if kind == "encoder":
        # a last-bit difference in a float moves an activation across a rounding boundary of the next per-tensor
        # 8-bit quantisation, and twelve layers pass that on
        return {"rel": 2e-2}
    if kind == "node":
        return {"rel": 1e-3}  # two TF32 convolutions: 11 significant bits
    # some fifty layers, every operand rounded to 11 (TF32) or 8 (bf16) significant bits: an accumulator that was
    # summed in another order rounds to the neighbouring operand now and then.  The normalisations of the generator
    # divide by small spreads and pass more of that on.
    if kind == "generator":
        return {"rel": 5e-3}
    return {"rel": 2e-2 if case["precision"] == "bf16" else 3e-3}


# ---- sessions ------------------------------------------------------------------------------------
_sessions = weakref.WeakValueDictionary()
_latest = [None]


def _build(case):
    kind = case["kind"]
    b = Session.builder()
    if case.get("graph"):
        b = b.with_cuda_graph(True)
    if kind == "cnn_f32":
        b = b.with_tuning(float_precision=case["precision"])
    if kind == "mlp":
        graph, weights, _, _ = models.build_int8_mlp(rows=case["rows"], dims=MLP_DIMS, spelling=case["spelling"])
        shapes = {"x": (case["rows"], MLP_DIMS[0])}
    elif kind == "cnn_int8":
        graph, weights, _, _ = models.build_resnet50_qlinear(batch=case["batch"], image=case["image"], typed_input=case["typed"])
        name = graph.input_names[0]
        shapes = {name: (case["batch"], 3, case["image"], case["image"])}
        if case["typed"]:
            b = b.with_input_types({name: np.uint8})
    elif kind == "cnn_f32":
        graph, weights, _, _ = models.build_resnet50_f32(batch=case["batch"], image=case["image"])
        shapes = {"input": (case["batch"], 3, case["image"], case["image"])}
    elif kind == "generator":
        graph, weights, _, _ = models.build_inswapper_f32(batch=case["batch"])
        shapes = {"target": (case["batch"], 3, 128, 128), "latent": (case["batch"], 512)}
    else:
        graph, weights, _, _ = models.build_bert_dynamic_int8(batch=case["batch"], seq=case["seq"], hidden=HIDDEN, heads=HEADS, ffn=FFN, layers=LAYERS,
                                                              vocab=VOCAB)
        shapes = {"input_ids": (case["batch"], case["seq"]), "attention_mask": (case["batch"], case["seq"])}
    session = b.with_input_shapes(shapes).build_from_graph(graph, weights)
    session.ensure_planned()
    return session


class _Block:
    """A context with the filters of a residual block registered, and the block's nodes."""

    def __init__(self, channels):
        rng = np.random.default_rng(channels)
        self.weights = {}
        for i in (1, 2):
            self.weights[f"w{i}"] = (rng.standard_normal((channels, channels, 3, 3)) * math.sqrt(2.0 / (9 * channels))).astype(np.float32)
            self.weights[f"b{i}"] = (rng.standard_normal(channels) * 0.1).astype(np.float32)
        self.ctx = CudaContext(0)
        self.ctx.register_weights(self.weights)
        pads = {"pads": [1, 1, 1, 1]}
        self.nodes = [Node("Conv", "conv1", ["x", "w1", "b1"], ["h"], dict(pads, activation="relu")), Node("Conv", "conv2", ["h", "w2", "b2"], ["r"], pads),
                      Node("Add", "add", ["r", "h"], ["y"], {})]


def _session(case):
    plan = {k: v for k, v in case.items() if k != "name"}
    if case["kind"] == "node":
        plan = {"kind": "node", "channels": case["channels"]}
    key = tuple(sorted(plan.items()))
    session = _sessions.get(key)
    if session is None:
        _latest[0] = None  # the one before goes first
        session = _Block(case["channels"]) if case["kind"] == "node" else _build(case)
        _sessions[key] = session
    _latest[0] = session
    return session


# ---- inputs --------------------------------------------------------------------------------------
def _inputs(case, gen):
    """Feeds of one batch, on the device."""
    kind = case["kind"]
    dev = {"device": "cuda", "generator": gen}
    if kind == "mlp":
        return {"x": torch.randn(case["rows"], MLP_DIMS[0], **dev)}
    b = case["batch"]
    if kind in ("cnn_int8", "cnn_f32"):
        x = torch.randn(b, 3, case["image"], case["image"], **dev)  # a normalised image
        if not case.get("typed"):
            return {"input": x}
        return {"input_q": torch.clamp(torch.round(x / (4.0 / 127.0)) + 128.0, 0, 255).to(torch.uint8)}
    if kind == "generator":
        z = torch.randn(b, 512, **dev)
        return {"target": torch.rand(b, 3, 128, 128, **dev), "latent": z / z.norm(dim=1, keepdim=True)}
    if kind == "encoder":
        s = case["seq"]
        ids = torch.randint(0, VOCAB, (b, s), **dev).float()
        lengths = torch.randint(max(1, s // 2), s + 1, (b, 1), **dev)  # sentences of a batch are padded to the longest
        lengths[0] = s
        return {"input_ids": ids, "attention_mask": (torch.arange(s, device="cuda")[None, :] < lengths).float()}
    return {"x": torch.randn(b, case["channels"], case["height"], case["width"], **dev)}


class State:
    def __init__(self, case, seed):
        self.session = _session(case)
        self.io = case.get("io", "node")
        gen = torch.Generator(device="cuda").manual_seed(seed)
        if self.io == "device":
            self.feeds = _inputs(case, gen)
            self.out_name = self.session.graph.output_names[0]
            self.out = torch.empty(_io_elements(case)[1], dtype=torch.float32, device="cuda")
        elif self.io == "stream":
            self.feeds = [{n: t.cpu().pin_memory().numpy() for n, t in _inputs(case, gen).items()} for _ in range(STREAM_BATCHES)]
        else:
            self.feeds = {n: t.cpu().numpy() for n, t in _inputs(case, gen).items()}
        torch.cuda.synchronize()  # the session has a stream of its own


def prepare(case, seed):
    return State(case, seed)


def run(state):
    s = state.session
    if state.io == "host":
        return s.run(state.feeds)
    if state.io == "stream":
        return s.run_pipelined(state.feeds)
    if state.io == "device":
        for name, t in state.feeds.items():
            s.bind_input_device(name, t.data_ptr(), np.uint8 if t.dtype == torch.uint8 else np.float32, t.numel())
        s.bind_output_device(state.out_name, state.out.data_ptr(), state.out.numel())
        s.run_with_binding(fetch=False)
        return state.out
    # one node at a time: the first convolution takes host lanes, the sum comes back to the host
    conv1, conv2, add = s.nodes
    h = try_cuda_dispatch_resident(conv1, s.weights, state.feeds, "device", s.ctx)
    r = try_cuda_dispatch_resident(conv2, s.weights, {"h": h}, "device", s.ctx)
    y = try_cuda_dispatch_resident(add, s.weights, {"r": r, "h": h, "__cap__": state.feeds["x"].size}, "host", s.ctx)[0]
    h.release()
    r.release()
    return y
