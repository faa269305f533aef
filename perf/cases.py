"""Performance cases: compiled routines as a user's program runs them.

Every case compiles a lowered routine (`backend.Code`), links it into a context (`Context.link`), turns
graph replay on as the benchmark and the data-parallel driver do, and runs it again and again on
buffers that stay on the GPU.  The routines are those of `ocannl_b200.workloads`:

  moons      half-moons MLP, one whole training step in single precision (forward, backprop, SGD)
  makemore   character MLP forward: embedding gather, tanh layer, log-softmax cross-entropy
  mlp        classifier forward: relu layers, softmax cross-entropy; 16-bit or single-precision weights
  train      the same classifier's training step through `Parallel.data_parallel` on one shard:
             forward + backprop, then plain or momentum SGD
  einsum     `b|m,k ; b|k,n => b|m,n`, bias and composed GELU
  decoder    decoder-only transformer forward: embedding, masked attention, layer norm, GELU FFN, head
  conv       convolution layer with bias, relu, squared error and all three gradients

`listed` holds the configurations of the repository's benchmark and smaller or ragged relatives of
them; `draw` takes the same routines over the range of sizes between a toy model and those.
"""
import math

import torch

from ocannl_b200 import backend as bk
from ocannl_b200 import parallel as par
from ocannl_b200 import workloads as W

STEPS = 4080          # length of the half-moons learning-rate schedule


def listed():
    return [
        # the smallest call: a 2-16-16-1 network on 20 points, one launch per step
        dict(name="moons_step_b20", kind="moons", batch=20, hid=16),
        # inference behind a request queue: whatever rows are waiting, here an odd handful
        dict(name="mlp_fwd_37_bf16", kind="mlp", rows=37, dims="784-1024-1024-10", prec="bfloat16"),
        # the benchmark's batch inference
        dict(name="mlp_fwd_8192_bf16", kind="mlp", rows=8192, dims="784-1024-1024-10", prec="bfloat16"),
        # a tutorial-sized language model evaluated over a batch, default (single) precision
        dict(name="makemore_4096_f32", kind="makemore", batch=4096, embed=10, hid=200, prec="single"),
        # batched contraction at its ordinary size
        dict(name="einsum_8x1024_bf16", kind="einsum", batch=8, m=1024, n=1024, k=1024, prec="bfloat16"),
        # the same spec over axes whose lengths come from data (classes, words, positions)
        dict(name="einsum_ragged_bf16", kind="einsum", batch=3, m=1000, n=777, k=333, prec="bfloat16"),
        # the largest: every SM full for most of a millisecond
        dict(name="einsum_8x4096_bf16", kind="einsum", batch=8, m=4096, n=4096, k=4096, prec="bfloat16"),
        # the benchmark's transformer, prompt evaluation of 64 full sequences
        dict(name="decoder_64x256_bf16", kind="decoder", batch=64, seq=256, layers=6, heads=8, d_head=64, d_model=512,
             d_ff=2048, nodes="local", prec="bfloat16"),
        # a few short sequences through a smaller model: 500 tokens, lengths off every tile size
        dict(name="decoder_5x100_bf16", kind="decoder", batch=5, seq=100, layers=4, heads=4, d_head=64, d_model=256,
             d_ff=1024, nodes="local", prec="bfloat16"),
        # the benchmark's training step
        dict(name="train_8192_bf16", kind="train", rows=8192, dims="784-1024-1024-10", prec="bfloat16", momentum=0.0),
        # a classic small classifier trained in default precision with Nesterov momentum
        dict(name="train_500_f32", kind="train", rows=500, dims="784-300-100-10", prec="single", momentum=0.9),
        # first convolution of an image classifier on 32 x 32 colour images, forward and backward
        dict(name="conv_64x32_f32", kind="conv", batch=64, size=32, cin=3, cout=32, kernel=3, stride=1, prec="single"),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread evenly over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _size(rng, lo, hi):
    """As `_log`; every other time a multiple of 8, as widths chosen by people tend to be."""
    v = _log(rng, lo, hi)
    return max(8, v // 8 * 8) if rng.random() < 0.5 and v >= 8 else v


def draw(rng):
    kind = rng.choice(["moons", "makemore", "mlp", "einsum", "einsum", "decoder", "train", "conv"])
    if kind == "moons":
        return dict(kind=kind, batch=_log(rng, 5, 512), hid=_size(rng, 8, 128))
    if kind == "makemore":
        return dict(kind=kind, batch=_log(rng, 32, 32768), embed=_log(rng, 4, 32), hid=_size(rng, 50, 512),
                    prec=rng.choice(["single", "bfloat16", "half"]))
    if kind in ("mlp", "train"):
        dims = "%d-%d-%d-%d" % (_size(rng, 32, 1024), _size(rng, 64, 2048), _size(rng, 64, 2048), _log(rng, 2, 64))
        c = dict(kind=kind, rows=_log(rng, 1 if kind == "mlp" else 16, 8192), dims=dims,
                 prec=rng.choice(["bfloat16", "bfloat16", "half", "single"]))
        if kind == "train":
            c["momentum"] = rng.choice([0.0, 0.9])
        return c
    if kind == "einsum":
        return dict(kind=kind, batch=_log(rng, 1, 8), m=_size(rng, 32, 4096), n=_size(rng, 32, 4096), k=_size(rng, 32, 4096),
                    prec=rng.choice(["bfloat16", "bfloat16", "half", "single"]))
    if kind == "decoder":
        heads, d_head = _log(rng, 1, 8), rng.choice([32, 64, 64])
        d_model = heads * d_head
        return dict(kind=kind, batch=_log(rng, 1, 64), seq=_size(rng, 8, 256), layers=rng.randint(1, 6), heads=heads, d_head=d_head,
                    d_model=d_model, d_ff=4 * d_model, nodes=rng.choice(["local", "local", "ctx"]), prec=rng.choice(["bfloat16", "half"]))
    return dict(kind=kind, batch=_log(rng, 1, 64), size=_size(rng, 8, 64), cin=_log(rng, 1, 32), cout=_size(rng, 8, 64),
                kernel=rng.choice([3, 3, 5]), stride=rng.choice([1, 1, 2]), prec=rng.choice(["single", "single", "bfloat16"]))


# ------------------------------------------------------------------ routines
def _dims(case):
    return tuple(int(v) for v in case["dims"].split("-"))


def _n_batches(case):
    return 1024 // case["batch"]


def _routines(case):
    """The lowered routine of a case; for a training step the update routine and the optimizer."""
    k = case["kind"]
    if k == "moons":
        return [W.moons_train_step(n_batches=_n_batches(case), batch=case["batch"], hid=case["hid"], steps=STEPS)]
    if k == "makemore":
        return [W.makemore_forward(batch=case["batch"], embed=case["embed"], hid=case["hid"], wprec=case["prec"])]
    if k == "mlp":
        return [W.mlp_forward(rows=case["rows"], dims=_dims(case), wprec=case["prec"])]
    if k == "train":
        return [W.mlp_train_update(rows=case["rows"], dims=_dims(case), wprec=case["prec"]),
                W.mlp_sgd(dims=_dims(case), wprec=case["prec"], momentum=case["momentum"],
                          weight_decay=1e-4 if case["momentum"] else 0.0, nesterov=case["momentum"] > 0.0)]
    if k == "einsum":
        return [W.einsum_gelu(case["batch"], case["m"], case["n"], case["k"], in_prec=case["prec"], y_prec=case["prec"])]
    if k == "decoder":
        return [W.transformer_forward(batch=case["batch"], seq=case["seq"], layers=case["layers"], d_model=case["d_model"],
                                      heads=case["heads"], d_head=case["d_head"], d_ff=case["d_ff"], wprec=case["prec"],
                                      attn_nodes=case["nodes"])]
    return [W.conv2d_update(batch=case["batch"], size=case["size"], cin=case["cin"], cout=case["cout"], kernel=case["kernel"],
                            stride=case["stride"], prec=case["prec"])]


# ------------------------------------------------------------------ inputs
def _one_hot(gen, shape):
    out = torch.zeros(shape, device="cuda")
    ids = torch.randint(0, shape[-1], shape[:-1], generator=gen, device="cuda")
    return out.scatter_(-1, ids.unsqueeze(-1), 1.0)


def _inputs(case, idents, gen):
    """{node: values} for everything a user fills: batches, weights, masks, rates."""
    k = case["kind"]

    def normal(shape, scale=1.0):
        return torch.randn(shape, generator=gen, device="cuda") * scale

    def uniform(shape, bound):
        return (torch.rand(shape, generator=gen, device="cuda") * 2.0 - 1.0) * bound

    out = {}
    if k == "moons":
        x, y = W.moons_inputs(n_points=1024, batch=case["batch"], seed=gen.initial_seed())
        out["moons_flat"], out["moons_classes"] = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
        for n in ("w1", "b1", "w2", "b2", "w3"):
            # U(-1, 1) at 16 hidden units; wider layers keep the same variance of a sum
            out[n] = uniform(idents[n], 1.0 if case["hid"] <= 16 else math.sqrt(16.0 / case["hid"]))
    elif k == "makemore":
        out["input_batch"] = torch.randint(0, 27, idents["input_batch"], generator=gen, device="cuda").float()
        out["target_batch"] = _one_hot(gen, idents["target_batch"])
        for n, fan in (("c", 27), ("w1", 3 * case["embed"]), ("b1", 3 * case["embed"]), ("w2", case["hid"]), ("b2", case["hid"])):
            out[n] = normal(idents[n], 1.0 / math.sqrt(fan))
    elif k in ("mlp", "train"):
        dims = _dims(case)
        out["x"], out["labels"] = normal(idents["x"]), _one_hot(gen, idents["labels"])
        for l, (n, b) in enumerate((("w1", "b1"), ("w2", "b2"), ("w_out", None))):
            bound = math.sqrt(6.0 / (dims[l] + dims[l + 1]))
            out[n] = uniform(idents[n], bound)
            if b:
                out[b] = uniform(idents[b], bound)
        if k == "train":
            out["learning_rate"] = torch.full((1,), 0.01, device="cuda")
    elif k == "einsum":
        # the spec's own scale: N(0, 1) operands
        out["a"], out["b"], out["bias"] = normal(idents["a"]), normal(idents["b"]), normal(idents["bias"])
    elif k == "decoder":
        out["tokens"] = _one_hot(gen, idents["tokens"])
        out["mask"] = torch.tril(torch.ones(idents["mask"], device="cuda"))
        for n, shape in idents.items():
            base = n.split("_", 1)[1] if n[0] == "l" and n[1].isdigit() else n
            if base in ("ln1_gamma", "ln2_gamma"):
                out[n] = torch.ones(shape, device="cuda")
            elif base in ("ln1_beta", "ln2_beta"):
                out[n] = torch.zeros(shape, device="cuda")
            elif base in ("tok_embed", "pos", "w_head", "w_q", "w_k", "w_v", "w_o", "ffn_w", "ffn_b", "ffn_w_out"):
                count = 1
                for d in shape:
                    count *= d
                fan_out = shape[0] * shape[1] if base in ("w_q", "w_k", "w_v") else shape[0]
                out[n] = normal(shape, math.sqrt(2.0 / (fan_out + count // fan_out)))
    else:
        out["x"], out["target"] = normal(idents["x"]), normal(idents["target"])
        out["kernel"] = normal(idents["kernel"], 1.0 / math.sqrt(case["kernel"] ** 2 * case["cin"]))
        out["bias"] = normal(idents["bias"], 0.1)
    return out


# ------------------------------------------------------------------ a linked program and its buffers
_TYPES = {"single": ("<f4", torch.float32), "half": ("<f2", torch.float16), "bfloat16": ("<i2", torch.bfloat16)}
_device = None


class _Program:
    """Compiled code, linked routines and the pools they are bound to; given back together."""

    def __init__(self, case):
        global _device
        if _device is None:
            _device = bk.Device(0)
        irs = _routines(case)
        if case["kind"] == "train":
            rep = par.DeviceReplica(_device, irs[0], irs[1], W.MLP_PARAM_NAMES)
            self.handle = par.DataParallel(rep, par.LocalExchange(), "mean", input_ident="x", target_ident="labels")
            self.codes, self.routines, self.context = [rep.update_code, rep.sgd_code], [rep.update, rep.sgd], rep.context
        else:
            code = bk.Code(irs[0])
            routine = bk.Context(_device).link(code)
            routine.use_graph(True)
            self.codes, self.routines, self.context = [code], [routine], routine.context
        self.written = {}
        for ir in irs:
            for t in ir.params():
                self.written[t.ident] = self.written.get(t.ident, False) or not t.read_only

    def __del__(self):
        if getattr(self, "context", None) is None:
            return
        _device.await_()
        for x in self.routines + self.codes:
            x.free()
        for pool in {p for p, _, _ in self.context.arrays.values()}:
            _device.free_pool(pool)
        self.context = None


class _Buffer:
    """A node's memory, for torch to look at; keeps the program that owns it."""

    def __init__(self, program, ident):
        pool, offset, t = program.context.arrays[ident]
        address, _ = _device.pool_address(pool)
        self.program = program
        self.__cuda_array_interface__ = {"shape": tuple(t.dims), "typestr": _TYPES[t.prec][0], "data": (address + offset, False),
                                         "version": 3, "strides": None}


def _view(program, ident):
    v = torch.as_tensor(_Buffer(program, ident), device="cuda")
    return v.view(_TYPES[program.context.arrays[ident][2].prec][1])


# what a decoder's caller looks at: the logits and each layer's projections and results
_DECODER_KEPT = ("q", "k", "v", "attn", "av", "x1", "ffn_h", "x2")


def _returned(case, program):
    names = [n for n, w in program.written.items() if w]
    if case["kind"] == "decoder":
        names = [n for n in names if n == "logits" or n.split("_", 1)[-1] in _DECODER_KEPT]
    return names


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.kind = case["kind"]
    s.program = _Program(case)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    nodes = s.program.context.arrays
    for ident, values in _inputs(case, {n: tuple(a[2].dims) for n, a in nodes.items()}, gen).items():
        _view(s.program, ident).copy_(values)
    torch.cuda.synchronize()
    s.outputs = {n: _view(s.program, n) for n in _returned(case, s.program)}
    s.routine = s.program.routines[0]
    s.handle = getattr(s.program, "handle", None)
    s.step = 0
    if s.kind == "moons":
        s.n_batches = _n_batches(case)
    return s


def run(s):
    if s.kind == "moons":
        # the next minibatch, the next point of the learning-rate schedule
        s.routine.run(i1=s.step % s.n_batches, i2=s.step % STEPS)
        s.step += 1
    elif s.handle is not None:
        s.handle.step()
    else:
        s.routine.run()
    return s.outputs


def work(case):
    """Bytes: every node the context holds crosses memory once, a node that is read and updated
    twice.  Operations: multiplications and additions of the contractions."""
    irs = _routines(case)
    nodes, updated = {}, set()
    for ir in irs:
        for t in ir.params():
            nodes[t.ident] = t.size_in_bytes
    if case["kind"] == "moons":
        updated = {"w1", "b1", "w2", "b2", "w3"}
        # of the data set one minibatch is read
        for n in ("moons_flat", "moons_classes"):
            nodes[n] //= _n_batches(case)
    elif case["kind"] == "train":
        updated = set(W.MLP_PARAM_NAMES) | {n for n in nodes if n.endswith("_sgd_momentum")}
    nbytes = sum(b * (2 if n in updated else 1) for n, b in nodes.items())
    k = case["kind"]
    if k == "moons":
        h = case["hid"]
        flops = 6.0 * case["batch"] * (2 * h + h * h + h)
    elif k == "makemore":
        flops = 2.0 * case["batch"] * case["hid"] * (3 * case["embed"] + 27)
    elif k in ("mlp", "train"):
        d = _dims(case)
        forward = 2.0 * case["rows"] * (d[0] * d[1] + d[1] * d[2] + d[2] * d[3])
        flops = forward if k == "mlp" else 3.0 * forward - 2.0 * case["rows"] * d[0] * d[1]
    elif k == "einsum":
        flops = 2.0 * case["batch"] * case["m"] * case["n"] * case["k"]
    elif k == "decoder":
        tokens, inner = case["batch"] * case["seq"], case["heads"] * case["d_head"]
        # a causal row attends to the positions up to its own
        flops = 2.0 * tokens * (case["layers"] * (4 * case["d_model"] * inner + 2 * case["d_model"] * case["d_ff"]
                                                  + inner * (case["seq"] + 1)) + 2 * 27 * case["d_model"])
    else:
        out = case["size"] if case["stride"] == 1 else (case["size"] - case["kernel"]) // case["stride"] + 1
        flops = 3.0 * 2.0 * case["batch"] * out * out * case["cout"] * case["kernel"] ** 2 * case["cin"]
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "moons" or (case["kind"] == "conv" and case["prec"] == "single"):
        return {"rel": 2e-5}        # sums of single-precision products in another order
    # 16-bit values between layers, or single-precision operands read as tf32: each rounds at 2^-9 to 2^-11,
    # and a value on the other side of a rounding boundary moves everything behind it
    return {"rel": 1e-2}
