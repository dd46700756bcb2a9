"""The calls that users of cospdnn_b200 make, as timed cases.

Three kinds of case, each one pass through the public entry points:

  layer    cospdnn_b200.layer(), the drop-in for one layer of the reference's
           host loop (feature-major activations, 16x16 blocks);
  prune    cospdnn_b200.prune_compact(), the pruning step of that loop;
  network  one batch through an Engine: set_input, run, result, and the final
           activations of the rows that survive (C entry
           cospdnn_engine_final_values into pinned memory that the program
           keeps).  The network, its weights and the engine are built once.

Weights and inputs are the package's seeded synthetic networks in the shapes
of the Graph Challenge (cospdnn_b200.synth): 32 weights of 1/16 per output,
XOR-mask patterns ("xor") or two dense 16x16 blocks per block column
("blocks"), binary input rows of density U[dlo, dhi).  Rows of low density die
within three layers; above a density of about 0.30 (1024 neurons), 0.35 (4096)
and 0.39 (16384) they live to the last layer.
"""
import ctypes as C

import numpy as np
import torch

import cospdnn_b200 as cs
from cospdnn_b200 import synth

PREC = {"fp32": cs.PREC_FP32, "fp16": cs.PREC_FP16, "bf16": cs.PREC_BF16}
#: input density from which a row lives through all layers, by width
LIVES = {1024: 0.30, 4096: 0.35, 16384: 0.39, 65536: 0.43}


def listed():
    def net(name, neuron, layers, rows, prec, dlo, dhi, weights="xor", given="bits", nets=1):
        return dict(name=name, kind="network", neuron=neuron, layers=layers, rows=rows, prec=prec, dlo=dlo, dhi=dhi,
                    weights=weights, given=given, nets=nets)

    return [
        # one 128-column tile of the smallest network: what is left is launch and latency
        dict(name="layer_1024_tile", kind="layer", neuron=1024, batch=128, weights="blocks", a="hilo", b="half"),
        # the reference's own call: 60000 images padded to its 128-column tile, reordered weights
        dict(name="layer_4096_batch", kind="layer", neuron=4096, batch=60032, weights="blocks", a="hilo", b="half"),
        # weights that were not reordered (about 30 blocks per column), FP32 data, a batch of odd size
        dict(name="layer_1024_ragged", kind="layer", neuron=1024, batch=9999, weights="xor", a="float", b="float"),
        # pruning after the first layers of a whole batch, half of the rows dead
        dict(name="prune_4096_batch", kind="prune", neuron=4096, batch=60000, keep=0.5, out="hilo"),
        # a few rows through the whole depth: a serving call
        net("net_1024_few_rows", 1024, 120, 64, "fp16", 0.25, 0.45),
        # the full-batch benchmark network in FP32
        net("net_1024_fp32", 1024, 120, 60000, "fp32", 0.08, 0.25),
        # rows that stay alive through all layers, as most do in the challenge's data
        net("net_1024_sustained", 1024, 120, 24000, "fp16", 0.25, 0.45, given="u8"),
        # the headline benchmark: 4096 neurons, the whole batch, FP16
        net("net_4096_batch", 4096, 120, 60000, "fp16", 0.08, 0.25),
        # reordered weights (dense blocks): the tensor-core path
        net("net_4096_blocks", 4096, 60, 60000, "fp16", 0.08, 0.25, weights="blocks"),
        # a wide network in BF16, a ragged part of a batch, some rows living on
        net("net_16384_bf16", 16384, 16, 6001, "bf16", 0.20, 0.41),
        # the widest network, one GPU's share of a batch
        net("net_65536_share", 65536, 4, 7500, "fp16", 0.10, 0.36),
        # several networks of several widths in one engine
        net("net_mix", 4096, 48, 12000, "fp16", 0.15, 0.38, nets=4),
    ]


def _log(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    kind = rng.choice(["layer", "layer", "prune", "network", "network", "network"])
    if kind == "layer":
        neuron = rng.choice([1024, 4096])
        weights = rng.choice(["blocks", "xor"])
        batch = _log(rng, 100, 60000 if weights == "blocks" else 30000 * 1024 // neuron)
        if rng.random() < 0.5:
            batch = (batch + 127) // 128 * 128  # as the reference pads it
        a = rng.choice(["hilo", "hilo", "float"])
        return dict(kind=kind, neuron=neuron, batch=batch, weights=weights, a=a, b="half" if a == "hilo" else "float")
    if kind == "prune":
        neuron = rng.choice([1024, 4096])
        return dict(kind=kind, neuron=neuron, batch=_log(rng, 200, 60000), keep=round(rng.uniform(0.05, 0.98), 3),
                    out=rng.choice(["hilo", "float"]))
    neuron = rng.choice([1024, 1024, 4096, 4096, 16384])
    layers = {1024: 120, 4096: 60, 16384: 12}[neuron]
    rows = _log(rng, 32, {1024: 30000, 4096: 20000, 16384: 5000}[neuron])
    weights = "blocks" if neuron == 4096 and rng.random() < 0.25 else "xor"
    dlo, dhi = rng.choice([(0.08, 0.25), (0.15, 0.40), (0.20, 0.42)])
    return dict(kind="network", neuron=neuron, layers=layers, rows=rows, prec=rng.choice(["fp16", "fp16", "bf16", "fp32"]),
                dlo=dlo, dhi=dhi, weights=weights, given=rng.choice(["bits", "u8", "f32"]), nets=1)


# ------------------------------------------------------------- one layer
def _masks(case, seed):
    f = synth.r1_masks if case["weights"] == "blocks" else synth.xor_masks
    return np.asarray(f(seed, 0, 0, case["neuron"]), np.int64)


def _bcsc(masks, neuron):
    """16x16 blocks of W[i][i ^ m] = 1/16: (col_ptr, row_index, values [blocks][16][16])."""
    high = np.unique(masks >> 4)
    pattern = np.zeros((len(high), 16, 16), np.float32)
    for m in masks:
        co = np.arange(16)
        pattern[np.searchsorted(high, m >> 4), co, co ^ (m & 15)] = 0.0625
    nb = neuron // 16
    at = np.arange(nb)[:, None] ^ high[None, :]
    order = np.argsort(at, axis=1)
    start = np.take_along_axis(at, order, 1) * 16
    return (np.arange(nb + 1, dtype=np.int32) * len(high), start.reshape(-1).astype(np.int32),
            pattern[order.reshape(-1)])


def _activations(neuron, batch, seed):
    """What one layer leaves: about half of the values 0, the others a few sixteenths less the bias."""
    g = torch.Generator("cuda").manual_seed(seed)
    x = torch.rand((neuron, batch), generator=g, device="cuda")
    return torch.where(x < 0.5, torch.zeros_like(x), x * 3.0)


def _prepare_layer(case, seed):
    n, batch = case["neuron"], case["batch"]
    cp, ri, v = _bcsc(_masks(case, seed), n)
    x = _activations(n, batch, seed)
    if case["a"] == "hilo":
        hi = x.half()
        a = torch.cat([hi, (x - hi.float()).half()])
    else:
        a = x
    flags = (cs.LAYER_A_FLOAT if case["a"] == "float" else 0) | (cs.LAYER_B_FLOAT if case["b"] == "float" else 0)
    b = torch.from_numpy(v).cuda()
    return dict(a=a, b=b if case["b"] == "float" else b.half(), c=torch.zeros((n, batch), device="cuda"),
                fuse=torch.arange(n, dtype=torch.int32, device="cuda"), cp=torch.from_numpy(cp).cuda(),
                ri=torch.from_numpy(ri).cuda(), flags=flags, bias=cs.BIAS[n])


def _run_layer(case, s):
    cs.layer(s["a"], s["b"], s["c"], s["fuse"], s["cp"], s["ri"], s["bias"], case["batch"], case["neuron"],
             flags=s["flags"], stream=torch.cuda.current_stream())
    return s["c"]


def _exact_layer(case, seed):
    n, batch = case["neuron"], case["batch"]
    x = _activations(n, batch, seed)
    if case["a"] == "hilo":
        hi = x.half()
        x = hi.double() + (x - hi.float()).half().double()
    y = _times_w(x.double().t().contiguous(), _masks(case, seed)).t()
    return (y + float(np.float32(cs.BIAS[n]))).clamp(0.0, 32.0)


def _times_w(y, masks):
    """y [rows][neuron] times W[i][i ^ m] = 1/16, in y's type."""
    j = torch.arange(y.shape[1], device=y.device)
    acc = torch.zeros_like(y)
    for m in masks:
        acc += y.index_select(1, j ^ int(m))
    return acc * 0.0625


# --------------------------------------------------------------- pruning
def _prepare_prune(case, seed):
    n, batch = case["neuron"], case["batch"]
    g = torch.Generator("cuda").manual_seed(seed)
    dead = torch.rand((1, batch), generator=g, device="cuda") >= case["keep"]
    c = _activations(n, batch, seed + 1).masked_fill_(dead, 0.0)
    pad = (batch + 127) // 128 * 128
    hilo = case["out"] == "hilo"

    def ints(k):
        return torch.zeros(k, dtype=torch.int32, device="cuda")

    return dict(c=c, out=torch.zeros(2 * n * pad if hilo else n * pad, dtype=torch.float16 if hilo else torch.float32,
                                     device="cuda"),
                category=ints(batch), map_in=torch.arange(batch, dtype=torch.int32, device="cuda"), map_out=ints(batch),
                count=ints(1), flags=cs.PRUNE_OUT_HALF_HILO if hilo else 0,
                ws=torch.empty(cs.prune_workspace_bytes(batch), dtype=torch.uint8, device="cuda"))


def _run_prune(case, s):
    cs.prune_compact(s["c"], case["neuron"], case["batch"], cs.THRESHOLD, s["out"], s["category"], s["map_in"],
                     s["map_out"], s["count"], s["ws"], flags=s["flags"], stream=torch.cuda.current_stream())
    return {k: s[k] for k in ("out", "category", "map_out", "count")}


# -------------------------------------------------------------- networks
def _nets(case):
    """(neuron, layers, rows) of each network of the case: the mix takes the widths 4096, 1024, 16384, 1024, ..."""
    out = []
    for k in range(case["nets"]):
        n = [case["neuron"], 1024, 16384, 1024][k % 4]
        rows = max(1, case["rows"] * 1024 // max(1024, n) + 37 * k)
        out.append((n, case["layers"] if n < 16384 else min(case["layers"], 12), rows))
    return out if case["nets"] > 1 else [(case["neuron"], case["layers"], case["rows"])]


def _weights(case, seed, k, neuron, layers):
    f = synth.r1_masks if case["weights"] == "blocks" else synth.xor_masks
    return [f(seed, k, l, neuron) for l in range(layers)]


def _inputs(case, seed, k, neuron, rows, given):
    x = synth.input_rows(rows, neuron, seed, net=k, dlo=case["dlo"], dhi=case["dhi"],
                         fmt=cs.INPUT_BITS if given == "bits" else cs.INPUT_U8)
    return x.float() if given == "f32" else x


def _live_share(case, neuron):
    return min(1.0, max(0.0, (case["dhi"] - LIVES[neuron]) / (case["dhi"] - case["dlo"])))


def _room(case, neuron, rows):
    """Rows of final activations that the program keeps memory for: more than live, a few kept rows at least."""
    return min(rows, int(1.4 * rows * _live_share(case, neuron)) + 64)


class _Program:
    """What a user's program keeps: the built engine, the batch, and pinned memory for the final activations."""

    def __init__(self, case, seed):
        self.nets, self.given = _nets(case), case["given"]
        self.engine = cs.Engine(torch.cuda.current_device())
        self.inputs, self.values = [], []
        for k, (n, layers, rows) in enumerate(self.nets):
            net = self.engine.add_net(n, layers, rows, precision=PREC[case["prec"]])
            for l, m in enumerate(_weights(case, seed, k, n, layers)):
                self.engine.set_layer_csc(net, l, *synth.masks_to_csc(m, n))
            self.inputs.append(_inputs(case, seed, k, n, rows, self.given))
            self.values.append(torch.zeros((_room(case, n, rows), n), pin_memory=True))
        self.engine.build()

    def batch(self):
        e, stream, out = self.engine, torch.cuda.current_stream(), []
        fmt = {"bits": cs.INPUT_BITS, "u8": cs.INPUT_U8, "f32": cs.INPUT_F32}[self.given]
        for net, x in enumerate(self.inputs):
            e.set_input(net, x, fmt=fmt, stream=stream)
        e.run(stream)
        for net, (_, _, rows) in enumerate(self.nets):
            r = e.result(net, stream)
            lives = np.zeros(rows, np.uint8)  # an answer for every row of the batch
            lives[r["categories"]] = 1
            v = self.values[net]
            if len(r["categories"]):
                rc = cs.lib().cospdnn_engine_final_values(e._h, net, C.cast(v.data_ptr(), C.POINTER(C.c_float)), len(v),
                                                          C.c_void_p(stream.cuda_stream))
                if rc != cs.OK:
                    raise cs.CospdnnError(rc, cs.lib().cospdnn_last_error().decode())
            out.append(dict(lives=lives, alive=r["alive"], values=v))
        return out


def _exact_network(case, seed):
    out = []
    for k, (n, layers, rows) in enumerate(_nets(case)):
        y = _inputs(case, seed, k, n, rows, "u8")
        bias, done = float(np.float32(cs.BIAS[n])), []
        step = max(1, (1 << 27) // n)  # rows at a time: 1 GB of doubles
        for lo in range(0, rows, step):
            part = y[lo:lo + step].double()
            for m in _weights(case, seed, k, n, layers):
                part = (_times_w(part, m) + bias).clamp_(0.0, 32.0)
                part = part[(part > cs.THRESHOLD).any(1)]
                if not len(part):
                    break
            done.append(part.cpu())
        kept, values = torch.cat(done), torch.zeros((_room(case, n, rows), n), dtype=torch.float64)
        values[:len(kept)] = kept[:len(values)]
        out.append(dict(lives=None, alive=None, values=values))
    return out


# ------------------------------------------------------------- interface
def prepare(case, seed):
    if case["kind"] == "layer":
        return case, _prepare_layer(case, seed)
    if case["kind"] == "prune":
        return case, _prepare_prune(case, seed)
    return case, _Program(case, seed)


def run(state):
    case, s = state
    if case["kind"] == "layer":
        return _run_layer(case, s)
    if case["kind"] == "prune":
        return _run_prune(case, s)
    return s.batch()


def work(case):
    if case["kind"] == "layer":
        n, batch = case["neuron"], case["batch"]
        blocks = (n // 16) * (2 if case["weights"] == "blocks" else 30)  # of 16x16 values
        return {"bytes": 8.0 * n * batch + blocks * 256 * (4 if case["b"] == "float" else 2), "flops": 2.0 * 32 * n * batch}
    if case["kind"] == "prune":
        n, batch = case["neuron"], case["batch"]
        return {"bytes": 4.0 * n * batch * (1 + case["keep"]) + 12.0 * batch, "flops": 1.0 * n * batch}
    total = {"bytes": 0.0, "flops": 0.0}
    for n, layers, rows in _nets(case):
        live = _live_share(case, n)
        given = {"bits": 0.125, "u8": 1.0, "f32": 4.0}[case["given"]]
        deep = layers if live else min(layers, 3)  # layers that some row reaches
        # inputs, two bytes per weight position of each layer reached, final rows; every other row is gone after two layers
        total["bytes"] += given * n * rows + 2.0 * 32 * n * deep + 4.0 * n * rows * live
        total["flops"] += 2.0 * 32 * n * rows * (2 + live * (deep - 2))
    return total


def exact(case, seed):
    if case["kind"] == "layer":
        return _exact_layer(case, seed)
    if case["kind"] == "prune":
        return None  # copies and splits: no computed values
    if case["neuron"] > 16384:
        return None
    return _exact_network(case, seed)
