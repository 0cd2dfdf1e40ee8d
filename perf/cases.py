"""The work a user of this framework has it do, as timed cases: whole optimised graphs (the benchmark networks), single
operators as the search times and the executor issues them, and the layout operators of the rewrites.

A case is a dict of plain values whose "kind" names the family:
  resnet18 / r3d18 / bert   a compiled graph of that network, one pass per run (pet_b200.graph.Graph.run)
  conv                      one 2-D convolution with its weights laid out once (Context.conv2d_run)
  matmul                    a product of two activations (Context.matmul), or with the second operand declared a weight once
                            (Context.matmul_run)
  banded                    banded self-attention: g2bmm -> softmax -> gbmml
  convtrans                 a transposed convolution, channels last, weights laid out once
  rewrite                   the transposes that PET's rewrites put before and after a convolution
Everything is fp32, the one data type of the operators.
"""
import functools
import math

import numpy as np
import torch

from pet_b200 import configs
from pet_b200.graph import Graph
from pet_b200.ops import Context

REWRITES = {"space_to_batch": configs.SPACE_TO_BATCH, "batch_to_space": configs.BATCH_TO_SPACE, "h2n": [configs.H2N],
            "n2h": [configs.N2H], "w2n": [configs.W2N], "n2w": [configs.N2W]}


def _conv(n, c, hw, f, k, stride=1, dil=1, groups=1, bias=True, act="none", residual=False, **more):
    return dict(kind="conv", n=n, c=c, hw=hw, f=f, k=k, stride=stride, dil=dil, groups=groups, bias=bias, act=act, residual=residual, **more)


def _matmul(b, m, n, k, trans_a=False, trans_b=False, weight=False, bias=False, act="none", **more):
    return dict(kind="matmul", b=b, m=m, n=n, k=k, trans_a=trans_a, trans_b=trans_b, weight=weight, bias=bias, act=act, **more)


def listed():
    return [
        # the smallest call: one 3x3 convolution of a ResNet block at batch 1 (benchmark configuration 1), where latency counts
        _conv(1, 64, 56, 64, 3, bias=False, name="conv3x3_64ch_56"),
        # a large single operator: the dilated convolution of benchmark configuration 2
        _conv(1, 512, 64, 512, 3, dil=2, bias=False, name="conv3x3_dilated_512ch_64"),
        # interactive image classification: the whole graph at batch 1 (benchmark configuration 3)
        dict(kind="resnet18", batch=1, size=224, classes=1000, name="resnet18_b1"),
        # the throughput workload of bench.py
        dict(kind="resnet18", batch=64, size=224, classes=1000, name="resnet18_b64"),
        # one clip through the video network (benchmark configuration 5)
        dict(kind="r3d18", batch=1, frames=16, size=112, classes=400, name="r3d18_b1"),
        # a sentence pair through the BERT-base encoder (benchmark configuration 4)
        dict(kind="bert", layers=12, seq=128, hidden=768, heads=12, ffn=3072, name="bert_base_seq128"),
        # the same encoder over a question-answering paragraph: more keys than the one-launch attention takes
        dict(kind="bert", layers=12, seq=384, hidden=768, heads=12, ffn=3072, name="bert_base_seq384"),
        # batched product of two activations at ragged sizes
        _matmul(4, 500, 1001, 770, name="matmul_b4_500x1001x770"),
        # one token against a large projection: bound by reading the weights
        _matmul(1, 1, 4096, 4096, weight=True, bias=True, name="matmul_m1_4096x4096"),
        # long-document attention at the one shape the reference ships its banded kernels for
        dict(kind="banded", b=1, n=10000, m=64, w=1000, dil=1, name="banded_attention_n10000_w1000"),
        # one up-sampling layer of an image generator
        dict(kind="convtrans", n=8, hw=32, f=128, c=64, k=4, stride=2, pad=1, bias=True, act="relu", name="convtrans4x4_s2_128_64_32"),
        # the layout step before a dilated convolution run as a dense one, at a batch
        dict(kind="rewrite", op="space_to_batch", n=16, c=512, h=64, w=64, name="space_to_batch_16x512x64x64"),
    ]


# ---- drawn cases ----------------------------------------------------------------------------------------------------------
def _log(rng, lo, hi):
    """A whole number of [lo, hi], spread evenly over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_conv(rng):
    k = rng.choice([1, 1, 3, 3, 3, 3, 5, 7])
    groups = rng.choice([1] * 9 + [2])
    c, f = _log(rng, 3, 512) if k == 7 or rng.random() < 0.3 else 8 * _log(rng, 1, 64), _log(rng, 16, 512)
    c, f = (c + groups - 1) // groups * groups, (f + groups - 1) // groups * groups
    stride = rng.choice([1, 1, 1, 2])
    return _conv(_log(rng, 1, 64), c, _log(rng, 7, 112), f, k, stride, 2 if k == 3 and stride == 1 and rng.random() < 0.2 else 1, groups,
                 rng.random() < 0.7, rng.choice(["none", "relu", "relu", "sigmoid", "tanh", "gelu"]), rng.random() < 0.3)


def _draw_matmul(rng):
    weight = rng.random() < 0.5
    b = 1 if weight else _log(rng, 1, 48)
    m = _log(rng, 1, 4096)
    four = 4 if rng.random() < 0.6 else 1
    return _matmul(b, m, four * _log(rng, 16 // four, 4096 // four), four * _log(rng, 16 // four, 4096 // four),
                   not weight and rng.random() < 0.15, rng.random() < 0.4, weight, rng.random() < 0.6,
                   rng.choice(["none", "none", "relu", "gelu"]))


def _draw_network(rng):
    kind = rng.choice(["resnet18", "resnet18", "bert", "bert", "r3d18"])
    if kind == "resnet18":
        return dict(kind=kind, batch=_log(rng, 1, 64), size=rng.randint(96, 256), classes=rng.randint(10, 1000))
    if kind == "r3d18":
        return dict(kind=kind, batch=rng.randint(1, 2), frames=rng.randint(8, 16), size=rng.randint(56, 128), classes=rng.randint(10, 400))
    hidden, heads = rng.choice([(768, 12), (512, 8), (1024, 16)])
    return dict(kind=kind, layers=rng.randint(1, 12), seq=_log(rng, 16, 512), hidden=hidden, heads=heads, ffn=4 * hidden)


def _draw_banded(rng):
    return dict(kind="banded", b=_log(rng, 1, 12), n=_log(rng, 512, 10000), m=rng.choice([32, 64, 64, 80]), w=_log(rng, 32, 1000),
                dil=rng.choice([1, 1, 1, 2, 4]))


def _draw_convtrans(rng):
    k, stride = rng.choice([(4, 2), (4, 2), (3, 1), (5, 2), (2, 2)])
    return dict(kind="convtrans", n=_log(rng, 1, 16), hw=_log(rng, 4, 64), f=4 * _log(rng, 4, 128), c=_log(rng, 3, 256), k=k, stride=stride,
                pad=(k - stride) // 2, bias=rng.random() < 0.7, act=rng.choice(["none", "relu", "tanh"]))


def _draw_rewrite(rng):
    op = rng.choice(sorted(REWRITES))
    n, h, w = _log(rng, 1, 32), 2 * _log(rng, 4, 56), 2 * _log(rng, 4, 56)
    return dict(kind="rewrite", op=op, n=4 * n if op in ("batch_to_space", "n2h", "n2w") else n, c=_log(rng, 16, 512), h=h, w=w)


def draw(rng):
    make = rng.choice([_draw_conv] * 3 + [_draw_matmul] * 3 + [_draw_network] * 3 + [_draw_banded, _draw_convtrans, _draw_rewrite])
    while True:
        case = make(rng)
        need = work(case)
        # a network: no more than the largest listed one; a single operator: no more than is ordinary for one
        if need["flops"] <= (2.2e11 if make is _draw_network else 4e10) and need["bytes"] <= 1.2e9:
            return case


# ---- what a user's program has in hand before the call ----------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _context():
    return Context(torch.cuda.current_device())


class _SeededInputs(configs.GraphBuilder):
    """A configuration with its own weights and the activations of one seed."""

    def __init__(self, graph, seed):
        super().__init__(graph)
        self.rng = np.random.default_rng(seed)

    def input(self, array):
        return super().input(self.rng.standard_normal(array.shape, np.float32))


class _DeviceView:
    """Lets torch read a tensor that a graph owns; keeps the graph, which frees its memory when it goes."""

    def __init__(self, graph, tensor):
        self.graph = graph
        self.__cuda_array_interface__ = {"shape": tuple(tensor.dims), "typestr": "<f4", "data": (int(graph.device_ptr(tensor)), False),
                                         "version": 3, "strides": None}


def _build_network(builder, case):
    kind = case["kind"]
    if kind == "resnet18":
        return configs.resnet18(builder, batch=case["batch"], size=case["size"], classes=case["classes"])
    if kind == "r3d18":
        return configs.r3d18(builder, batch=case["batch"], frames=case["frames"], size=case["size"], classes=case["classes"])
    return configs.bert_encoder(builder, layers=case["layers"], seq=case["seq"], hidden=case["hidden"], heads=case["heads"], ffn=case["ffn"])


def _out_extent(size, k, stride, dil, pad):
    return (size - (k - stride) * dil + 2 * pad) // stride


def prepare(case, seed):
    ctx, kind = _context(), case["kind"]
    state = {"ctx": ctx, "case": case}
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, scale=1.0):
        return torch.randn(shape, device="cuda", generator=gen) * scale

    if kind in ("resnet18", "r3d18", "bert"):
        graph = Graph(ctx)
        builder = _SeededInputs(graph, seed)
        out = _build_network(builder, case)
        graph.setOutputs([out])
        graph.compile()
        builder.load()
        state["graph"] = graph
        state["out"] = torch.as_tensor(_DeviceView(graph, out), device=ctx.device)
    elif kind == "conv":
        n, c, hw, f, k, cpg = case["n"], case["c"], case["hw"], case["f"], case["k"], case["c"] // case["groups"]
        pad = case["dil"] * (k - 1) // 2
        state["x"] = normal(n, c, hw, hw)
        state["bias"] = normal(f) if case["bias"] else None
        state["plan"] = ctx.conv2d_plan((n, c, hw, hw), (f, cpg, k, k), pad, pad, case["stride"], case["stride"], case["dil"], case["dil"],
                                        case["bias"], case["act"])
        ctx.conv2d_set_weights(state["plan"], normal(f, cpg, k, k, scale=math.sqrt(2.0 / (cpg * k * k))))
        state["residual"] = normal(*state["plan"].out_shape) if case["residual"] else None
    elif kind == "matmul":
        b, m, n, k = case["b"], case["m"], case["n"], case["k"]
        ashape, bshape = (b, k, m) if case["trans_a"] else (b, m, k), (b, n, k) if case["trans_b"] else (b, k, n)
        state["a"], state["b"] = normal(*ashape), normal(*bshape, scale=1.0 / math.sqrt(k))
        state["bias"] = normal(n) if case["bias"] else None
        if case["weight"]:
            state["plan"] = ctx.matmul_plan(ashape, bshape, case["trans_a"], case["trans_b"], case["bias"], case["act"])
            ctx.matmul_set_weights(state["plan"], state["b"])
    elif kind == "banded":
        b, n, m = case["b"], case["n"], case["m"]
        state["q"], state["k"], state["v"] = normal(b, n, m, scale=1.0 / math.sqrt(m)), normal(b, n, m), normal(b, n, m)
    elif kind == "convtrans":
        n, hw, f, c, k = case["n"], case["hw"], case["f"], case["c"], case["k"]
        state["x"] = normal(n, hw, hw, f)
        state["bias"] = normal(c) if case["bias"] else None
        state["plan"] = ctx.convtrans_plan((n, hw, hw, f), (k, k, f, c), case["pad"], case["pad"], case["stride"], case["stride"],
                                           bias=case["bias"], act=case["act"])
        ctx.convtrans_run(state["plan"], state["x"], normal(k, k, f, c, scale=math.sqrt(2.0 / (k * k * f))), state["bias"])
    else:
        state["x"] = normal(case["n"], case["c"], case["h"], case["w"])
    return state


# ---- one pass -----------------------------------------------------------------------------------------------------------------
def run(state):
    ctx, case = state["ctx"], state["case"]
    kind = case["kind"]
    if kind in ("resnet18", "r3d18", "bert"):
        state["graph"].run()
        return state["out"]
    if kind == "conv":
        return ctx.conv2d_run(state["plan"], state["x"], state["bias"], residual=state["residual"])
    if kind == "matmul":
        if case["weight"]:
            return ctx.matmul_run(state["plan"], state["a"], None, state["bias"])
        return ctx.matmul(state["a"], state["b"], case["trans_a"], case["trans_b"], state["bias"], case["act"])
    if kind == "banded":
        scores = ctx.g2bmm(state["q"], state["k"], case["w"], case["dil"])
        return ctx.gbmml(ctx.softmax(scores), state["v"], case["dil"])
    if kind == "convtrans":
        return ctx.convtrans_run(state["plan"], state["x"], None, state["bias"])
    return ctx.transpose_chain(state["x"], REWRITES[case["op"]])


# ---- what a pass cannot do without --------------------------------------------------------------------------------------------
class _Counter:
    """Walks a network's layers with shapes alone: multiply-adds of its contractions, words of its weights."""

    def __init__(self):
        self.macs = self.weights = self.ends = 0

    def layer(self, outputs, k, filters, per_filter):
        self.macs += outputs * k
        self.weights += filters * per_filter + filters
        return self

    def work(self):
        return {"bytes": 4.0 * (self.weights + self.ends), "flops": 2.0 * self.macs}


def _residual_net(case):
    """ResNet-18 and its 3-D form: stem, four stages of two blocks, classifier."""
    count, video, batch = _Counter(), case["kind"] == "r3d18", case["batch"]
    hw, depth, taps = _out_extent(case["size"], 7, 2, 1, 3), case.get("frames", 1), 27 if video else 9
    stem = 3 * 49 * (3 if video else 1)
    count.layer(batch * depth * hw * hw * 64, stem, 64, stem)
    count.ends = batch * (3 * depth * case["size"] ** 2 + case["classes"])
    cin = 64
    if not video:
        hw = _out_extent(hw, 3, 2, 1, 1)
    for stage, cout in enumerate((64, 128, 256, 512)):
        for block in range(2):
            stride = 2 if stage > 0 and block == 0 else 1
            hw = _out_extent(hw, 3, stride, 1, 1)
            depth = _out_extent(depth, 3, stride, 1, 1) if video else depth
            outputs = batch * depth * hw * hw * cout
            count.layer(outputs, cin * taps, cout, cin * taps).layer(outputs, cout * taps, cout, cout * taps)
            if stride != 1 or cin != cout:
                count.layer(outputs, cin, cout, cin)
            cin = cout
    return count.layer(batch * case["classes"], cin, case["classes"], cin).work()


def _encoder(case):
    count, seq, hidden, ffn = _Counter(), case["seq"], case["hidden"], case["ffn"]
    count.ends = 2 * seq * hidden
    for _ in range(case["layers"]):
        for cin, cout in ((hidden, hidden),) * 4 + ((hidden, ffn), (ffn, hidden)):
            count.layer(seq * cout, cin, cout, cin)
        count.macs += 2 * seq * seq * hidden
    return count.work()


def work(case):
    kind = case["kind"]
    if kind in ("resnet18", "r3d18"):
        return _residual_net(case)
    if kind == "bert":
        return _encoder(case)
    if kind == "conv":
        n, c, hw, f, k, cpg = case["n"], case["c"], case["hw"], case["f"], case["k"], case["c"] // case["groups"]
        out = n * f * _out_extent(hw, k, case["stride"], case["dil"], case["dil"] * (k - 1) // 2) ** 2
        return {"bytes": 4.0 * (n * c * hw * hw + f * cpg * k * k + out * (2 if case["residual"] else 1)), "flops": 2.0 * out * cpg * k * k}
    if kind == "matmul":
        b, m, n, k = case["b"], case["m"], case["n"], case["k"]
        return {"bytes": 4.0 * b * (m * k + k * n + m * n), "flops": 2.0 * b * m * n * k}
    if kind == "banded":
        b, n, m, bw = case["b"], case["n"], case["m"], 2 * case["w"] + 1
        # three calls with results of their own: the band is written and read twice (scores, probabilities)
        return {"bytes": 4.0 * b * (4 * n * bw + 4 * n * m), "flops": 4.0 * b * n * bw * m}
    if kind == "convtrans":
        n, hw, f, c, k, st = case["n"], case["hw"], case["f"], case["c"], case["k"], case["stride"]
        out = (hw - 1) * st - 2 * case["pad"] + k
        return {"bytes": 4.0 * (n * hw * hw * f + k * k * f * c + n * out * out * c), "flops": 2.0 * n * hw * hw * k * k * f * c}
    return {"bytes": 8.0 * case["n"] * case["c"] * case["h"] * case["w"], "flops": 0.0}


def tolerance(case):
    """Layout operators move words.  A single contraction with fp32 operands and fp32 sums: 1e-5.  A network compounds its
    layers' rounding, each followed by a normalisation or a residual sum."""
    if case["kind"] == "rewrite":
        return "exact"
    return {"rel": 3e-5 if case["kind"] in ("resnet18", "r3d18", "bert") else 1e-5}
