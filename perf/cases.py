"""Performance cases: what a program that uses this framework has it do, through its public entry points.

A case is one network of `kyanite_b200.configs` at one batch size and one way of calling the executor:

    io "host"    `CudaExecutor.evaluate(inputs)`: arrays of the caller in, fresh arrays out, one call after the other
    io "pair"    two executors of the network on one GPU, `evaluate_begin` on both, then `evaluate_end` on both, as a
                 host does that keeps a GPU busy while it fills and reads batches
    io "device"  `run_async` on inputs that are on the GPU already; results stay on the GPU

An executor is built once for a network and batch size and is kept, as a program that serves requests keeps it; the
weights belong to it.  What changes from one state to the next, by the seed, is the network's input.
"""
import functools
import math

import numpy as np
import torch

from kyanite_b200 import configs
from kyanite_b200.executor import MATH_F32, MATH_TF32, CudaExecutor
from kyanite_b200.graph import DType, OpKind

# ------------------------------------------------------------------------------------------------ the cases

MLP = {"net": "mlp"}
TOWER = {"net": "tower", "channels": 128, "blocks": 16, "board": 8}
BERT = {"net": "bert", "layers": 12, "hidden": 768, "heads": 12}
DECODER = {"net": "decoder", "layers": 1, "d_model": 4096, "heads": 32, "ffn": 11008}
UNET = {"net": "unet", "levels": 2}


def _case(arch, batch, io, math_mode="tf32", **more):
    return {**arch, "batch": batch, "io": io, "math": math_mode, **more}


def listed():
    return [
        # the smallest call: a small policy network asked for a handful of states at a time
        {"name": "mlp_b8", **_case(MLP, 8, "host")},
        # one position, as a player at the board asks for it: the answer's latency counts
        {"name": "tower_b1", **_case(TOWER, 1, "host")},
        # the usual batch of a self-play server, one call after the other
        {"name": "tower_b256", **_case(TOWER, 256, "host")},
        # the same server with two batches in flight
        {"name": "tower_b256_pair", **_case(TOWER, 256, "pair")},
        # the largest batch of the usual sweep, batches produced on the GPU
        {"name": "tower_b2048_device", **_case(TOWER, 2048, "device")},
        # another game: 9 x 9 board, narrower network, a batch that is no multiple of anything
        {"name": "tower_9x9_b101", **_case({**TOWER, "channels": 64, "blocks": 8, "board": 9}, 101, "host")},
        # exact f32 arithmetic, for reproducing results of another implementation
        {"name": "tower_f32_b64", **_case(TOWER, 64, "host", "f32")},
        # one short sentence through the encoder: latency over many small steps
        {"name": "bert_b1_s120", **_case(BERT, 1, "host", seq=120)},
        # the encoder's largest batch, ids produced and embeddings used on the GPU
        {"name": "bert_b32_s512_device", **_case(BERT, 32, "device", seq=512)},
        # a prompt of full length through a decoder layer with half storage
        {"name": "decoder_f16_s2048", **_case(DECODER, 1, "device", seq=2048, dtype="f16")},
        # a short prompt of ragged length
        {"name": "decoder_f16_s333", **_case(DECODER, 1, "host", seq=333, dtype="f16")},
        # one denoising step on one latent
        {"name": "unet_b1_device", **_case(UNET, 1, "device", size=64)},
    ]


def _spread(rng, low, high):
    """A whole number from low to high, spread over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    while True:
        net = rng.choice(["mlp", "tower", "tower", "tower", "bert", "bert", "decoder", "decoder", "unet"])
        io = rng.choice(["host", "host", "device"])
        if net == "mlp":
            case = _case(MLP, _spread(rng, 1, 4096), io)
        elif net == "tower":
            arch = {"net": "tower", "channels": rng.choice([64, 128, 128, 256]), "blocks": rng.choice([4, 8, 16]),
                    "board": rng.choice([7, 8, 8, 9])}
            mode = rng.choice(["tf32", "tf32", "tf32", "f32"])
            case = _case(arch, _spread(rng, 1, 2048), rng.choice([io, "pair"]), mode)
        elif net == "bert":
            arch = {"net": "bert", "layers": rng.choice([4, 6, 12]), **rng.choice([{"hidden": 384, "heads": 6}, {"hidden": 768, "heads": 12}])}
            case = _case(arch, _spread(rng, 1, 32), io, seq=_spread(rng, 16, 512))
        elif net == "decoder":
            arch = rng.choice([DECODER, {"net": "decoder", "layers": 2, "d_model": 2048, "heads": 16, "ffn": 5504}])
            case = _case(arch, rng.choice([1, 1, 2, 3]), io, seq=_spread(rng, 32, 2048), dtype=rng.choice(["f16", "f16", "f32"]))
        else:
            case = _case(UNET, rng.choice([1, 2, 3]), io, size=8 * _spread(rng, 3, 8))
        if _cost(case) * (2 if case["io"] == "pair" else 1) <= _cost(_case(BERT, 32, "device", seq=512)):
            return case


def _cost(case):
    """About the multiply-adds of a pass, exact f32 ones counted at what they cost outside the tensor cores."""
    if case["net"] == "mlp":
        return 1e4 * case["batch"]
    if case["net"] == "tower":
        area = case["board"] ** 2
        return 18.0 * case["blocks"] * case["batch"] * area * case["channels"] ** 2 * (20 if case["math"] == "f32" else 1)
    rows = case["batch"] * case.get("seq", 0)
    if case["net"] == "bert":
        return case["layers"] * rows * case["hidden"] * (12.0 * case["hidden"] + 2 * case["seq"])
    if case["net"] == "decoder":
        d = case["d_model"]
        return case["layers"] * rows * d * (4.0 * d + 3 * case["ffn"] + 2 * case["seq"])
    return 1e11 * case["batch"] * (case["size"] / 64.0) ** 2


# ------------------------------------------------------------------------------------------------ their networks


@functools.lru_cache(maxsize=1)
def _network(key):
    """(graph, make_inputs) of a case's network; the weights are the configuration's own, from its fixed seed."""
    a = dict(key)
    if a["net"] == "mlp":
        return configs.mlp()
    if a["net"] == "tower":
        return configs.resnet_tower(channels=a["channels"], blocks=a["blocks"], board=a["board"])
    if a["net"] == "bert":
        return configs.bert_encoder(layers=a["layers"], hidden=a["hidden"], heads=a["heads"], ffn=4 * a["hidden"], seq=a["seq"])
    if a["net"] == "decoder":
        return configs.llama_decoder(layers=a["layers"], d_model=a["d_model"], heads=a["heads"], ffn=a["ffn"], vocab=1000,
                                     seq=a["seq"], dtype=DType.F16 if a["dtype"] == "f16" else DType.F32)
    widths = (320, 640, 1280)[:a["levels"]]
    return configs.unet_step(levels=widths, res_blocks=1, attention_levels=tuple(range(a["levels"])), size=a["size"])


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "batch", "io", "math")))


_kept = {}


def _executors(case):
    """The executors that a program would keep for this network and batch size (those of the latest case)."""
    key = (_key(case), case["batch"], case["io"], case["math"])
    if key not in _kept:
        for old in [e for group in _kept.values() for e in group]:
            old.close()
        _kept.clear()
        graph, _ = _network(_key(case))
        blob = graph.to_bytes()
        mode = MATH_F32 if case["math"] == "f32" else MATH_TF32
        _kept[key] = [CudaExecutor(0, blob, case["batch"], math_mode=mode) for _ in range(2 if case["io"] == "pair" else 1)]
    return _kept[key]


class _DeviceArray:
    """An executor's device buffer as torch sees it."""

    def __init__(self, executor, is_output, index):
        array = (executor.host_outputs if is_output else executor.host_inputs)[index]
        pointer, _ = executor.device_buffer(is_output, index)
        self.__cuda_array_interface__ = {"shape": array.shape, "typestr": array.dtype.str, "data": (pointer, False), "version": 3}


def prepare(case, seed):
    executors = _executors(case)
    _, make_inputs = _network(_key(case))
    sets = [make_inputs(case["batch"], 1 + 1000 * seed + k) for k in range(len(executors))]
    state = {"io": case["io"], "executors": executors, "inputs": sets}
    if case["io"] == "device":
        ex = executors[0]
        state["stream"] = torch.cuda.ExternalStream(ex.stream())
        state["inputs"] = [torch.from_numpy(x).cuda() for x in sets[0]]
        state["device_inputs"] = [torch.as_tensor(_DeviceArray(ex, False, i), device="cuda") for i in range(len(ex.host_inputs))]
        state["device_outputs"] = [torch.as_tensor(_DeviceArray(ex, True, i), device="cuda") for i in range(len(ex.host_outputs))]
    return state


def run(state):
    executors, inputs = state["executors"], state["inputs"]
    if state["io"] == "host":
        return executors[0].evaluate(inputs[0])
    if state["io"] == "pair":
        for ex, x in zip(executors, inputs):
            ex.evaluate_begin(x)
        return [ex.evaluate_end() for ex in executors]
    with torch.cuda.stream(state["stream"]):
        for to, x in zip(state["device_inputs"], inputs):
            to.copy_(x, non_blocking=True)
    executors[0].run_async()
    return state["device_outputs"]


# ------------------------------------------------------------------------------------------------ what a pass needs


@functools.lru_cache(maxsize=None)
def _needs(key, batch):
    """(bytes, flops) of one pass: inputs, weights and outputs once each; multiply-adds of convolutions and matmuls."""
    graph, make_inputs = _network(key)
    dims = lambda v: [d.eval(batch) for d in graph[v].shape]  # noqa: E731
    values = graph.all_values()
    bytes_, flops = float(sum(x.nbytes for x in make_inputs(batch, 0))), 0.0
    looked_up = set()
    for v in values:
        info = graph[v]
        if info.kind == OpKind.MATMUL:
            b, m, n = dims(v)
            flops += 2.0 * b * m * n * dims(values[info.inputs[0]])[2]
        elif info.kind == OpKind.CONV:
            flops += 2.0 * math.prod(dims(v)) * math.prod(dims(values[info.inputs[1]])[1:])
        elif info.kind == OpKind.GATHER and graph[values[info.inputs[0]]].kind == OpKind.CONSTANT:
            looked_up.add(info.inputs[0])  # of a table no more is read than the rows that are looked up
            bytes_ += math.prod(dims(v)) * info.dtype.size_bytes
    for i, v in enumerate(values):
        if graph[v].kind == OpKind.CONSTANT and i not in looked_up:
            bytes_ += graph[v].tensor.nbytes
    bytes_ += sum(math.prod(dims(v)) * graph[v].dtype.size_bytes for v in graph.outputs)
    return bytes_, flops


def work(case):
    bytes_, flops = _needs(_key(case), case["batch"])
    times = 2 if case["io"] == "pair" else 1
    return {"bytes": times * bytes_, "flops": times * flops}


def tolerance(case):
    if case.get("dtype") == "f16":
        return {"rel": 5e-3}  # every value stored with 11 bits, a few dozen roundings in a row
    if case["math"] == "tf32":
        return {"rel": 2e-3}  # operands of contractions rounded to 11 bits, sums in f32
    return {"rel": 1e-5}
