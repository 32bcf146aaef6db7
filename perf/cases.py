"""The work users of this package have it do, as measurable cases: what a program holds before the call (`prepare`), the
call itself through the public entry points (`run`), the work it cannot do without (`work`) and how far two correct
implementations may differ (`tolerance`).

Kinds of cases
  infer     a batch of coordinates through a network, on the GPU (FusedNetwork under no_grad with fp32 tables, or the
            Network class with the fp16 tables a trainer leaves behind)
  host      the same for a batch that lives in page-locked host memory (Network.inference_host)
  train     one step of FusedTrainer: forward, L2 loss, backward, Adam
  autograd  FusedNetwork inside a user's own PyTorch loss: forward, mse_loss, backward
  encode    a stand-alone FusedEncoding in front of the user's own layers, forward and backward

The networks are the benchmark configurations of the package (qmlp/configs.py); table sizes vary at run time.
"""
import math
import os
import sys

sys.path.insert(0, os.path.abspath("quick-mlp_b200"))

import torch  # noqa: E402

import qmlp  # noqa: E402
from qmlp import configs  # noqa: E402
from qmlp.bindings import Network, QuickMLP  # noqa: E402

NETWORKS = {
    "tiny": lambda c: configs.config1(),
    "mlp": lambda c: configs.config2(),
    "grid3d": lambda c: configs.config3(log2_hashmap_size=c["log2_rows"]),
    "mixed": lambda c: configs.config4(log2_hashmap_size=c["log2_rows"]),
    "grid4d": lambda c: configs.config5(log2_hashmap_size=c["log2_rows"]),
}
# range of the coordinates and the table sizes (log2 of the rows of a hashed level) a network is used with
LOW = {"tiny": 0.0, "mlp": -1.0, "grid3d": 0.0, "mixed": 0.0, "grid4d": 0.0}
ROWS = {"grid3d": (14, 19), "mixed": (14, 18), "grid4d": (16, 22)}

ENCODINGS = {
    # a dense feature pyramid over an image, five resolutions of four features
    "pyramid2d": dict(n_in=2, n_levels=5, n_features=4, log2_hashmap_size=-1, min_resolution=16, max_resolution=256),
    # a small hash grid over a volume, eight levels of two features
    "hash3d": dict(n_in=3, n_levels=8, n_features=2, log2_hashmap_size=10, min_resolution=4, max_resolution=512, per_level_scale=2.0),
}


def listed():
    return [
        # a picker or a single ray bundle: a thousand points through the plain MLP, where only latency counts
        dict(name="mlp_infer_1k", kind="infer", net="mlp", table="float", log2_rows=0, points=1000),
        # a full frame or volume slab through the plain MLP
        dict(name="mlp_infer_4m", kind="infer", net="mlp", table="float", log2_rows=0, points=1 << 22),
        # the same network called by a program whose points live on the host
        dict(name="mlp_infer_host_1m", kind="host", net="mlp", table="float", log2_rows=0, points=1 << 20),
        # rendering from a trained hash grid, fp16 tables
        dict(name="grid3d_infer_half_1m", kind="infer", net="grid3d", table="half", log2_rows=19, points=1 << 20),
        # an odd-sized set of query points against the module's own fp32 tables
        dict(name="grid3d_infer_float_100k", kind="infer", net="grid3d", table="float", log2_rows=19, points=100003),
        # a time-varying volume with tables far larger than the L2 cache
        dict(name="grid4d_infer_half_16m", kind="infer", net="grid4d", table="half", log2_rows=22, points=1 << 24),
        # the training step of the package's headline benchmark
        dict(name="grid3d_train_1m", kind="train", net="grid3d", table="half", log2_rows=19, points=1 << 20),
        # a small training batch, interactive fitting
        dict(name="grid3d_train_8k", kind="train", net="grid3d", table="half", log2_rows=19, points=8191),
        # two encodings of four features, uneven layer widths, several outputs
        dict(name="mixed_train_2m", kind="train", net="mixed", table="half", log2_rows=18, points=1 << 21),
        # image fitting or a PDE residual in a user's own loop: weight and coordinate gradients of the plain MLP
        dict(name="mlp_autograd_64k", kind="autograd", net="mlp", table="float", log2_rows=0, points=64000, input_grad=True),
        # a hash grid trained by a user's own loop: weight and table gradients
        dict(name="grid3d_autograd_256k", kind="autograd", net="grid3d", table="float", log2_rows=19, points=1 << 18, input_grad=False),
        # image features in front of the user's own layers: forward, and the gradient of the feature tables
        dict(name="pyramid_encode_1m", kind="encode", net="pyramid2d", table="float", log2_rows=0, points=1000003, input_grad=False),
    ]


def _points(rng, low, high):
    """log-uniform, every other one a multiple of 64, the rest odd or ragged"""
    n = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    return max(low, n // 64 * 64) if rng.random() < 0.4 else min(n | 1, high)


def draw(rng):
    kind = rng.choice(["infer", "infer", "infer", "host", "train", "train", "autograd", "autograd", "encode"])
    if kind == "infer":
        net = rng.choice(["tiny", "mlp", "grid3d", "mixed", "grid4d"])
        c = dict(kind=kind, net=net, table="float" if net in ("tiny", "mlp") else rng.choice(["half", "float"]))
        high = {"tiny": 1 << 22, "mlp": 1 << 22, "grid3d": 1 << 21, "mixed": 1 << 21, "grid4d": 1 << 22}[net]
        c["points"] = _points(rng, 256, high)
    elif kind == "host":
        c = dict(kind=kind, net="mlp", table="float", points=_points(rng, 1 << 14, 1 << 22))
    elif kind == "train":
        net = rng.choice(["grid3d", "mixed"])
        c = dict(kind=kind, net=net, table=rng.choice(["half", "half", "float"]), points=_points(rng, 1 << 11, 1 << 20))
    elif kind == "autograd":
        net = rng.choice(["mlp", "grid3d", "mixed"])
        c = dict(kind=kind, net=net, table="float", points=_points(rng, 1 << 10, 1 << 19), input_grad=rng.random() < 0.5)
    else:
        c = dict(kind=kind, net=rng.choice(["pyramid2d", "hash3d"]), table="float", points=_points(rng, 1 << 12, 1 << 21),
                 input_grad=rng.random() < 0.5)
    c["log2_rows"] = rng.randint(*ROWS[c["net"]]) if c["net"] in ROWS else 0
    return c


# ---- inputs and parameters -------------------------------------------------------------------------------------------
def _uniform(gen, shape, low, high, dtype=torch.float32):
    return torch.empty(shape, dtype=dtype, device="cuda").uniform_(low, high, generator=gen)


def _weights(gen, network, cfg):
    """Xavier-uniform weights and small biases on the unpadded entries, fp16; the padding is zero."""
    w = torch.zeros((network.num_network_parameters(),), dtype=torch.float32, device="cuda")
    n_in = sum(network.encoding(i).num_output_channels() for i in range(network.num_encodings()))
    for i, layer in enumerate(cfg["network"]):
        n_out = layer["n_out"]
        bound = math.sqrt(6.0 / (n_in + n_out))
        network.parameter_view(i, False, w)[:n_out, :n_in] = _uniform(gen, (n_out, n_in), -bound, bound)
        if layer["bias"]:
            network.parameter_view(i, True, w)[:n_out] = _uniform(gen, (n_out,), -0.05, 0.05)
        n_in = n_out
    return w.half()


def _target(x, channels):
    """smooth functions of the coordinates, one per output channel"""
    return torch.stack([torch.sin((8 + 2 * k) * x[:, 0]) * torch.cos(6 * x[:, 1]) * torch.sin((4 + k) * x[:, 2])
                        for k in range(channels)], dim=1).contiguous()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    torch.manual_seed(seed)
    QuickMLP.set_log_level("error")
    n = case["points"]
    if case["kind"] == "encode":
        enc = qmlp.FusedEncoding(configs.dumps(configs.hashgrid(**ENCODINGS[case["net"]])))
        count = enc._encoding.parameter_count()
        x = _uniform(gen, (n, ENCODINGS[case["net"]]["n_in"]), 0.0, 1.0)
        if case["input_grad"]:
            x.requires_grad_(True)
        table = _uniform(gen, (count,), -0.5, 0.5).requires_grad_(True)
        grad = _uniform(gen, (n, enc.num_output_channels()), -1.0, 1.0)
        return dict(kind="encode", encoding=enc, x=x, table=table, grad=grad)

    cfg = NETWORKS[case["net"]](case)
    x = _uniform(gen, (n, cfg["num_inputs"]), LOW[case["net"]], 1.0)
    if case["kind"] == "autograd" or (case["kind"] == "infer" and case["table"] == "float"):
        # weight gradients in fp32 for training, fp16 weights (the module's default) for inference
        train = case["kind"] == "autograd"
        net = qmlp.FusedNetwork(configs.dumps(cfg), weight_dtype=torch.float32 if train else torch.float16)
        with torch.no_grad():
            net.weights.copy_(_weights(gen, net._network, cfg))
            for p in net.encoding_parameters:
                if p.requires_grad:
                    p.uniform_(-0.5, 0.5, generator=gen)
        if not train:
            return dict(kind="infer", call=net, x=x)
        t = _target(x, cfg["num_outputs"])
        if case["input_grad"]:
            x.requires_grad_(True)
        leaves = [net.weights] + [p for p in net.encoding_parameters if p.requires_grad] + ([x] if case["input_grad"] else [])
        return dict(kind="autograd", net=net, x=x, target=t, leaves=leaves)

    net = Network(configs.dumps(cfg))
    weights = _weights(gen, net, cfg)
    grids = [net.encoding(i) for i in range(net.num_encodings())]
    if case["kind"] == "train":
        # a run in progress: trained-looking tables, and Adam moments of the size the gradients have
        tr = qmlp.FusedTrainer(net, grid_half_copy=case["table"] == "half")
        master, m, v = (torch.zeros_like(tr.master) for _ in range(3))
        tr.segment(master, 0).copy_(weights)
        sizes = [1e-3] + [0.1 / n] * len(grids)
        for i, s in enumerate(sizes):
            if i > 0:
                tr.segment(master, i).uniform_(-0.1, 0.1, generator=gen)
            tr.segment(m, i).normal_(0.0, 0.1 * s, generator=gen)
            tr.segment(v, i).fill_(s * s)
        tr.load_state_dict(dict(master=master, adam_m=m, adam_v=v, step=100))
        return dict(kind="train", trainer=tr, x=x, target=_target(x, cfg["num_outputs"]))
    tables = [_uniform(gen, (g.parameter_count(),), -0.5, 0.5, torch.float16) if g.has_parameters() else None for g in grids]
    if case["kind"] == "host":
        x = x.cpu().pin_memory()
        out = torch.empty((n, cfg["num_outputs"]), dtype=torch.float32, pin_memory=True)
        return dict(kind="host", net=net, x=x, weights=weights, tables=tables, out=out)
    return dict(kind="infer", call=lambda p: net.inference(p, weights, tables), x=x)


def run(state):
    kind = state["kind"]
    if kind == "infer":
        with torch.no_grad():
            return state["call"](state["x"])
    if kind == "host":
        return state["net"].inference_host(state["x"], state["weights"], state["tables"], output=state["out"])
    if kind == "train":
        tr = state["trainer"]
        tr.step(state["x"], state["target"])
        return [tr.master, tr.adam_m, tr.adam_v, tr.half, tr.loss_sum]
    if kind == "autograd":
        for p in state["leaves"]:
            p.grad = None
        out = state["net"](state["x"])
        loss = torch.nn.functional.mse_loss(out, state["target"])
        loss.backward()
        return [out.detach(), loss.detach()] + [p.grad for p in state["leaves"]]
    state["x"].grad = state["table"].grad = None
    out = state["encoding"](state["x"], state["table"])
    out.backward(state["grad"])
    return [out.detach(), state["table"].grad] + ([state["x"].grad] if state["x"].requires_grad else [])


# ---- what the work amounts to ----------------------------------------------------------------------------------------
def _level_rows(g):
    """rows of every level of a grid description (the level table of the package: floor(resolution) per level)"""
    d, levels = g["n_in"], g["n_levels"]
    lo, hi = g["min_resolution"], g["max_resolution"]
    scale = g.get("per_level_scale") or (math.exp(math.log(hi / lo) / (levels - 1)) if levels > 1 else 1.0)
    cap = 1 << g["log2_hashmap_size"] if g["log2_hashmap_size"] >= 0 else None
    rows = [int(lo * scale ** i + 1e-6) ** d for i in range(levels)]
    return [min(r, cap) if cap else r for r in rows]


def work(case):
    n, kind = case["points"], case["kind"]
    if kind == "encode":
        grids, cfg = [dict(ENCODINGS[case["net"]])], None
        n_in, n_out = grids[0]["n_in"], grids[0]["n_levels"] * grids[0]["n_features"]
    else:
        cfg = NETWORKS[case["net"]](case)
        grids = [dict(n_in=e["n_in"], n_levels=e["n_levels"], n_features=e["n_features_per_level"],
                      log2_hashmap_size=e["log2_hashmap_size"], min_resolution=e["min_resolution"], max_resolution=e["max_resolution"],
                      per_level_scale=e.get("per_level_scale")) for e in cfg["encodings"] if e["id"] == "HashGrid"]
        n_in, n_out = cfg["num_inputs"], cfg["num_outputs"]
    elem = 2 if case["table"] == "half" else 4
    all_rows = touched = 0.0     # table elements, and those that this many points reach at most
    blend = 0.0                  # multiply-adds of the interpolation
    for g in grids:
        for r in _level_rows(g):
            all_rows += r * g["n_features"]
            touched += min(r, n << g["n_in"]) * g["n_features"]
        blend += n * g["n_levels"] * (1 << g["n_in"]) * g["n_features"] * 2
    layers = 0.0
    if cfg is not None:
        width = sum(g["n_levels"] * g["n_features"] for g in grids) or n_in
        for l in cfg["network"]:
            layers += 2.0 * n * width * l["n_out"]
            width = l["n_out"]
    io = 4.0 * n * (n_in + n_out)
    if kind in ("infer", "host"):
        return {"bytes": io + touched * elem, "flops": layers + blend}
    if kind == "train":      # every parameter: master, both moments read and written, the half copy written
        return {"bytes": io + touched * elem + all_rows * 26, "flops": 3 * layers + 2 * blend}
    grad_in = 4.0 * n * n_in if case["input_grad"] else 0.0
    out_twice = 4.0 * n * n_out      # outputs written by the forward call, their adjoints read by the backward call
    return {"bytes": io + out_twice + grad_in + touched * 4 + all_rows * 4, "flops": 3 * layers + 2 * blend}


def tolerance(case):
    if case["kind"] == "encode":
        # fp32 throughout; the cell fraction of a position at resolution R carries a rounding error of R * 2^-24
        return {"rel": 1e-4}
    if case["kind"] in ("infer", "host"):
        # every layer's output is rounded to fp16 (2^-11) and its accumulation order is free
        return {"rel": 5e-3}
    # fp16 activations, deltas and loss gradients; a pre-activation within one fp16 rounding of zero may take the other
    # branch of a relu
    return {"rel": 1e-2, "max": 0.5}
