"""Performance cases of the NCN layer: what a user of the package has it do, over the range of sizes.

Each case goes through the package's public surface (the reference's module and function names):

  heads   NCNNetCuda on [B, N, E] tokens with several heads of features: training step or forward only
  rows    NCNNetCuda (or RefInvTorchNaive, the reversible stack) with one feature per position
  stack   NCNResidualStack: residual layers, each a net of several stages
  padded  fused_ncn_cuda_ctxlen stage by stage: a context length per batch row
  host    net_fwd_bwd_host: activations in pinned host memory, results back in pinned host memory

A training step is the forward and the gradients of both streams' inputs and of every weight, as in the
middle of a model: x and dy are drawn from N(0, 1), the second stream and its cotangent are smaller.
"""
import math

import torch

import ncn_cuda_b200 as ncn
from ncn_cuda_b200.host import net_fwd_bwd_host

ALPHA = 0.9


def _heads(name, B, N, E, heads, n, stages, dtype="f32", act="tanh", train=True):
    return {"name": name, "kind": "heads", "B": B, "N": N, "E": E, "heads": heads, "n": n, "stages": stages,
            "dtype": dtype, "act": act, "train": train}


def _rows(name, B, N, n, stages, dtype="f32", act="tanh", train=True, mode="auto", w_var=0.0):
    return {"name": name, "kind": "rows", "B": B, "N": N, "n": n, "stages": stages, "dtype": dtype, "act": act,
            "train": train, "mode": mode, "w_var": w_var or 1.0 / n}


def listed():
    return [
        # The shape of the reference's own gradient test: four sequences of 256 tokens, 128 features in 4 heads, groups of
        # 32, 3 stages.  The smallest training step: launches and host work count.
        _heads("tokens_4", 4, 256, 128, 4, 32, 3),
        # The same model at a training batch (bench.py's ref_e128 shape, a quarter of its rows).
        _heads("tokens_1024", 1024, 256, 128, 4, 32, 3),
        # A wider model in mixed precision: bf16 activations, fp32 weights, groups of 16.
        _heads("tokens_bf16", 64, 512, 256, 8, 16, 4, dtype="bf16"),
        # The CPU-sized layer: 1024 rows of 1024 positions, groups of 2, 10 stages.  4 MB per tensor.
        _rows("rows_1024_g2", 1024, 1024, 2, 10),
        # The layer the headline benchmark is quoted on: 65536 rows of 4096 positions, groups of 4, 6 stages.
        _rows("rows_65536_g4", 65536, 4096, 4, 6),
        # Forward only (inference, or a frozen layer) with the linear activation, at an ordinary batch.
        _rows("rows_infer_linear", 16384, 4096, 4, 6, act="linear", train=False),
        # bf16 storage, rows of 8192 positions, groups of 16 (a quarter of the benchmark's rows).
        _rows("rows_bf16_g16", 65536, 8192, 16, 4, dtype="bf16", w_var=1.0 / 16),
        # The reversible stack: the backward rebuilds every activation from the output (benchmark shape, a quarter of its rows).
        _rows("rows_invert_g8", 32768, 4096, 8, 4, mode="invert", w_var=0.01),
        # Ragged: 1000 rows of 3000 positions, neither a power of two.
        _rows("rows_ragged", 1000, 3000, 4, 5),
        # One GPU's share of the 12-layer residual stack in bf16.  The largest.
        {"name": "stack_12", "kind": "stack", "B": 131072, "N": 2048, "n": 8, "layers": 12, "stages": 4, "dtype": "bf16", "act": "tanh"},
        # A padded batch: 64 sequences of up to 256 tokens, each with its own length; the token model above.
        {"name": "padded_64", "kind": "padded", "B": 64, "N": 256, "E": 128, "heads": 4, "n": 32, "stages": 3, "act": "tanh"},
        # The headline layer for a caller whose activations live on the host.
        {"name": "host_8192", "kind": "host", "B": 8192, "N": 4096, "n": 4, "stages": 6, "act": "tanh"},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _batch(rng, lo, hi, per_row, steps, cap):
    """Rows for a number of elements drawn over its logarithm, with elements * steps bounded by `cap`."""
    return max(1, int(min(_log(rng, lo, hi), cap / steps) / per_row))


def draw(rng):
    kind = rng.choice(["heads", "heads", "heads", "rows", "rows", "rows", "rows", "stack", "padded", "host"])
    act = rng.choice(["tanh", "tanh", "tanh", "tanh", "linear", "relu", "sigmoid"])
    if kind in ("heads", "padded"):
        n = rng.choice([4, 8, 16, 32])
        d = rng.choice([8, 16, 32, 32, 64, 24, 48] if kind == "heads" else [16, 32, 32, 24])
        heads = rng.choice([1, 2, 3, 4, 8])
        N = n * rng.randint(3, 32)  # odd numbers of groups among them
        stages = rng.randint(1, 4)
        case = {"kind": kind, "B": 0, "N": N, "E": d * heads, "heads": heads, "n": n, "stages": stages}
        if kind == "padded":
            case["act"] = rng.choice(["tanh", "linear"])
            case["B"] = _batch(rng, 1 << 16, 1 << 22, N * d * heads, n * stages, 2e8)
            return case
        case["dtype"] = rng.choice(["f32", "f32", "bf16"])
        case["act"] = rng.choice([act, act, act, act, "leaky-relu"])
        case["train"] = rng.random() < 0.75
        case["B"] = _batch(rng, 1 << 16, 1 << 25, N * d * heads, n * stages, 3e9)
        return case
    n = rng.choice([2, 4, 8, 16])
    if rng.random() < 0.5:
        N = 2 ** rng.randint(9, 13)
    else:
        N = 8 * int(_log(rng, 30, 700))  # any multiple of 8 elements that the groups divide
        N -= N % max(8, n)
    stages = rng.randint(2, 10 if n == 2 else 6 if n == 4 else 4)
    if kind == "rows":
        dtype = rng.choice(["f32", "f32", "bf16"])
        mode = rng.choice(["auto", "auto", "auto", "invert"]) if dtype == "f32" and n * stages <= 32 else "auto"
        case = {"kind": kind, "B": 0, "N": N, "n": n, "stages": stages, "dtype": dtype, "act": "tanh" if mode == "invert" else act,
                "train": mode == "invert" or rng.random() < 0.75, "mode": mode, "w_var": 0.01 if mode == "invert" else 1.0 / n}
        case["B"] = _batch(rng, 1 << 13, 1 << 28, N, n * stages, 1e10)
        return case
    if kind == "stack":
        layers = rng.randint(2, 12)
        case = {"kind": kind, "B": 0, "N": 2 ** rng.randint(9, 12), "n": rng.choice([4, 8]), "layers": layers, "stages": rng.randint(2, 4),
                "dtype": rng.choice(["bf16", "bf16", "f32"]), "act": "tanh"}
        case["B"] = _batch(rng, 1 << 16, 1 << 27, case["N"], layers * case["n"] * case["stages"], 3e10)
        return case
    case = {"kind": "host", "B": 0, "N": N, "n": n, "stages": stages, "act": act}
    case["B"] = _batch(rng, 1 << 18, 1 << 25, N, n * stages, 3e9)
    return case


def _steps(case):
    """Recurrence steps that every element goes through."""
    return case["n"] * case["stages"] * case.get("layers", 1)


def work(case):
    elems = case["B"] * case["N"] * case.get("E", 1)
    w = 2 if case.get("dtype") == "bf16" else 4
    train = case.get("train", True)
    # in: x, xa (and both cotangents); out: y, ya (and both input gradients); the weights are a few KB
    weights = 4 * 2 * case.get("E", 1) * case["stages"] * case.get("layers", 1)
    bytes_ = elems * w * (8 if train else 4) + weights * (2 if train else 1)
    # operations per element and step: forward 7 with the scale factors of the decay carried outside the steps (T = x P + Q, the
    # activation, a += c F, x += c a), 2 more for the dot product over a head's features; backward 18 (the inverse
    # of a step, its activation again, the cotangents and the weight sums), 8 more over features
    features = case.get("E", 1) > 1
    ops = (9 if features else 7) + ((26 if features else 18) if train else 0)
    return {"bytes": bytes_, "flops": elems * _steps(case) * ops}


def tolerance(case):
    if case.get("dtype") == "bf16":
        # each residual layer of a stack rounds its result to bf16 again
        return {"rel": 2e-2 if case["kind"] == "stack" else 1e-2}
    if "relu" in case["act"]:
        # the derivative jumps at 0: rounding flips the sign of a few pre-activations (about 1e-7 of them in each step), and
        # each one changes its element's gradient by a few per cent
        return {"rel": 3e-4, "max": 0.3}
    # fp32; a reversible walk over more than 16 steps multiplies earlier rounding by 1/0.9 per step
    chain = case["n"] if case["kind"] == "padded" else _steps(case) if case.get("mode") == "invert" else 0
    return {"rel": 2e-5 if chain > 16 else 1e-5}


def _dtype(case):
    return torch.bfloat16 if case.get("dtype") == "bf16" else torch.float32


def _weights(case, g, var):
    layers = (case["layers"],) if case["kind"] == "stack" else ()
    return torch.randn(*layers, case["stages"], 2 * case.get("E", 1), generator=g, device="cuda") * math.sqrt(var)


def _net(case, W):
    E, heads, stages = case.get("E", 1), case.get("heads", 1), case["stages"]
    if case.get("mode") == "invert":
        ws = [w.clone().requires_grad_(True) for w in W]
        return ncn.RefInvTorchNaive(ALPHA, case["act"], stages, case["n"], heads, ws), ws
    if case["act"] == "leaky-relu":  # the activation that only the reversible surface names
        ws = [w.clone().requires_grad_(True) for w in W]
        return ncn.RefInvTorchNaive(ALPHA, "leaky-relu", stages, case["n"], heads, ws), ws
    if case["kind"] == "stack":
        net = ncn.NCNResidualStack(case["layers"], ALPHA, case["act"], case["n"], heads, stages, E).cuda()
        with torch.no_grad():
            net.weight.copy_(W)
        return net, [net.weight]
    net = ncn.NCNNetCuda(ALPHA, case["act"], case["n"], heads, stages, E).cuda()
    with torch.no_grad():
        for mod, w in zip(net.ncn_modules, W):
            mod.weight.copy_(w)
    return net, list(net.parameters())


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (case["B"], case["N"], case.get("E", 1))

    def randn(scale=1.0):
        return torch.randn(shape, generator=g, device="cuda", dtype=_dtype(case)).mul_(scale)

    if case["kind"] == "host":
        def pinned(scale):
            t = torch.empty(shape, dtype=torch.float32, pin_memory=True)
            t.copy_(randn(scale))
            return t

        s = {"case": case, "x": pinned(1.0), "xa": pinned(0.25), "dy": pinned(1.0), "dya": pinned(0.25)}
        s["out"] = tuple(torch.empty(shape, dtype=torch.float32, pin_memory=True) for _ in range(4))
        s["W"] = _weights(case, g, 1.0 / case["n"])
        return s
    train = case.get("train", True)
    s = {"case": case, "x": randn().requires_grad_(train), "xa": randn(0.25).requires_grad_(train)}
    if train:
        s["dy"], s["dya"] = randn(), randn(0.25)
    var = case.get("w_var") or (1.0 / (case["E"] // case["heads"]) if "E" in case else 1.0 / case["n"])
    W = _weights(case, g, var)
    if case["kind"] == "padded":
        s["ws"] = [w.clone().requires_grad_(True) for w in W]
        s["ctxlen"] = torch.randint(1, case["N"] + 1, (case["B"],), generator=g, device="cuda", dtype=torch.int32)
    else:
        s["net"], s["ws"] = _net(case, W)
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "host":
        return net_fwd_bwd_host(s["x"], s["xa"], s["W"], s["dy"], s["dya"], ALPHA, case["act"], case["n"], 1, out=s["out"])
    if case["kind"] == "padded":
        y, ya = s["x"], s["xa"]
        act = ncn.ops.ACTIVATION_CODES[case["act"]]
        for l, w in enumerate(s["ws"]):
            y, ya = ncn.fused_ncn_cuda_ctxlen(y, ya, w, s["ctxlen"], ALPHA, act, case["n"], case["heads"], l)
    elif not case.get("train", True):
        with torch.no_grad():
            return s["net"](s["x"], s["xa"])
    else:
        y, ya = s["net"](s["x"], s["xa"])
    grads = torch.autograd.grad((y, ya), (s["x"], s["xa"], *s["ws"]), (s["dy"], s["dya"]))
    return (y.detach(), ya.detach(), *grads)
